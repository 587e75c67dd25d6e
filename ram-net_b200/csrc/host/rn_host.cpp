// Native host path of ramnet_ops: the public calls in their common form, from Python arguments to kernel launches.
//
// A decode step is one kernel of about ten microseconds and the small prefill and training shapes are a few such
// kernels, while the Python front end (validation, axis moves, broadcasting, operator dispatch, argument marshalling)
// takes 150 us per decode call, 300 us per prefill and 1 ms per forward and backward pass.  This module takes the calls
// that need none of that generality: plain CUDA tensors in the (B, T, H, ...) layout, nothing to broadcast but the
// positions, a float32 state or none.  Everything else, and every call that has something wrong with it, is
// declined (None), and the Python front end then handles it as before, with its own checks and messages.  Declined as
// well: tensor subclasses, dispatch and function modes, functorch transforms and tracing, which need the registered
// operators.
//
//   attention(...)   random_access_memory_attention (packages/ramnet-ops/src/ramnet_ops/ram_attn.py:106-367 of the
//                    reference): decode step, prefill, and prefill under autograd (RamAttention below)
//   topk_addr(...)   topk_addr (ram_attn.py:46-103), without autograd
//   workspace(...)   the scratch buffer of a (device, stream), shared with the Python operators
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <mutex>
#include <optional>
#include <utility>

#include "../../../include/ramnet_b200.h"

namespace {

using at::Tensor;

void check(int rc) {
    TORCH_CHECK(rc == 0, rn_last_error());
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return RN_F32;
        case at::kHalf: return RN_F16;
        case at::kBFloat16: return RN_BF16;
        default: return -1;
    }
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, at::Device device) {
    return Tensor(at::detail::empty_cuda(size, type, device, std::nullopt));
}

// ---- what a call has to look like --------------------------------------------------------------------------------
// Nothing may want to see the operators underneath: dispatch / function modes, functorch layers, tracers.
bool plain_context() {
    if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled()) return false;
    static const c10::DispatchKeySet watching({c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                               c10::DispatchKey::FuncTorchDynamicLayerBackMode, c10::DispatchKey::Functionalize,
                                               c10::DispatchKey::PythonDispatcher, c10::DispatchKey::Tracer,
                                               c10::DispatchKey::FuncTorchVmapMode});
    const auto tls = c10::impl::tls_local_dispatch_key_set();
    return !tls.included_.has_any(watching) && !tls.excluded_.has(c10::DispatchKey::AutogradCUDA);
}

bool plain_tensor(PyObject *o, Tensor *out) {
    if (!THPVariable_CheckExact(o)) return false;
    const Tensor &t = THPVariable_Unpack(o);
    static const c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::Negative,
                                              c10::DispatchKey::Conjugate, c10::DispatchKey::ZeroTensor,
                                              c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                              c10::DispatchKey::BatchedNestedTensor});
    if (!t.is_cuda() || t.layout() != at::kStrided || t.key_set().has_any(special) || t._fw_grad(0).defined()) return false;
    *out = t;
    return true;
}

bool take_int(PyObject *o, int64_t *v) {
    if (!PyLong_Check(o)) return false;
    *v = PyLong_AsLongLong(o);
    if (*v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}
bool take_float(PyObject *o, double *v) {
    if (PyFloat_Check(o)) {
        *v = PyFloat_AS_DOUBLE(o);
        return true;
    }
    int64_t i;
    if (!take_int(o, &i)) return false;
    *v = double(i);
    return true;
}
// a value or a two-item tuple / list of values
template <typename V, typename F>
bool take_pair(PyObject *o, V *a, V *b, F take) {
    if (take(o, a)) {
        *b = *a;
        return true;
    }
    if (PyTuple_Check(o) && PyTuple_GET_SIZE(o) == 2) return take(PyTuple_GET_ITEM(o, 0), a) && take(PyTuple_GET_ITEM(o, 1), b);
    if (PyList_Check(o) && PyList_GET_SIZE(o) == 2) return take(PyList_GET_ITEM(o, 0), a) && take(PyList_GET_ITEM(o, 1), b);
    return false;
}

struct Positions {
    Tensor t;  // undefined: the token index
    int kind = RN_POS_INDEX;
    int64_t strides[2] = {0, 0};
    const void *ptr() const { return t.defined() ? t.const_data_ptr() : nullptr; }
};
// positions (B,T) or (1,T), int32 or int64
bool take_positions(PyObject *o, int64_t B, int64_t T, at::Device device, Positions *p) {
    if (o == Py_None) return true;
    if (!plain_tensor(o, &p->t) || p->t.device() != device || p->t.dim() != 2) return false;
    if (p->t.size(1) != T || (p->t.size(0) != B && p->t.size(0) != 1)) return false;
    if (p->t.scalar_type() == at::kInt) p->kind = RN_POS_I32;
    else if (p->t.scalar_type() == at::kLong) p->kind = RN_POS_I64;
    else return false;
    p->strides[0] = p->t.size(0) == 1 ? 0 : p->t.stride(0);
    p->strides[1] = p->t.stride(1);
    return true;
}

// Every batch row (and its single token) one contiguous block of what follows: the form the decode kernels read.
bool contiguous_rows(const Tensor &t, int64_t *ld) {
    int64_t inner = 1;
    for (int64_t d = t.dim() - 1; d >= 2; --d) {
        if (t.size(d) != 1 && t.stride(d) != inner) return false;
        inner *= t.size(d);
    }
    *ld = t.size(0) == 1 ? inner : t.stride(0);
    return *ld >= inner;
}

struct Call {
    int64_t B, T, H, U, P, A, C, E, Kw, Kr;
    double rho_w, rho_r, eps, mass_init;
    bool mass_aware;
    int code;  // dtype code of logits, values, gates
    at::Device device{at::kCUDA, 0};
    Positions pos;
    Tensor mask;  // undefined: no mask
    const uint8_t *mask_ptr() const { return mask.defined() ? static_cast<const uint8_t *>(mask.const_data_ptr()) : nullptr; }
};

constexpr int64_t INT_LIMIT = (int64_t(1) << 31) - 1;

// ---- scratch -----------------------------------------------------------------------------------------------------
// One buffer per (device, stream), grown on demand and handed back by release(): calls on one stream are ordered, so
// they may share it, and every call rewrites what it later reads.  Used with the GIL held, from taking the buffer to
// the last launch that uses it, so two threads on one stream cannot interleave; the lock guards the table itself.  A
// stream capture takes its buffer from the capturing allocator and keeps nothing here.
std::mutex g_ws_lock;
std::map<std::pair<int, cudaStream_t>, Tensor> &ws_table() {
    static auto *table = new std::map<std::pair<int, cudaStream_t>, Tensor>();  // never destroyed: outlives the allocator
    return *table;
}
Tensor workspace(at::Device device, cudaStream_t stream, int64_t bytes) {
    bytes = std::max<int64_t>(bytes, 256);
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return empty({bytes}, at::kByte, device);
    std::lock_guard<std::mutex> lock(g_ws_lock);
    Tensor &t = ws_table()[{device.index(), stream}];
    if (!t.defined() || t.numel() < bytes) {
        t = Tensor();  // given back first: the two need not exist side by side
        t = empty({bytes}, at::kByte, device);
    }
    return t;
}

// ---- the calls ---------------------------------------------------------------------------------------------------
void swap_axes(const Tensor &t, int64_t (&s)[5]) {  // (B,T,H,U,P) -> strides over (B,H,U,P,T)
    s[0] = t.stride(0); s[1] = t.stride(2); s[2] = t.stride(3); s[3] = t.stride(4); s[4] = t.stride(1);
}
struct Rows {  // (B,T,H,C) -> strides over (B,H,T,C); (B,T,H) -> over (B,H,T)
    int64_t s[4];
    explicit Rows(const Tensor &t) : s{t.stride(0), t.stride(2), t.stride(1), t.dim() == 4 ? t.stride(3) : 1} {}
};

struct Decoded {
    Tensor idx, val;  // (B,T,H,Kw+Kr)
    int64_t s[4];     // strides over (B,H,K,T)
};

Decoded decode_addresses(const Call &c, const Tensor &w, const Tensor &r, cudaStream_t stream) {
    const int64_t K = c.Kw + c.Kr;
    Decoded d{empty({c.B, c.T, c.H, K}, at::kInt, c.device), empty({c.B, c.T, c.H, K}, at::kFloat, c.device),
              {c.T * c.H * K, K, 1, c.H * K}};
    int64_t sa[5];
    swap_axes(w, sa);
    check(rn_addr_fwd_pos(w.const_data_ptr(), r.const_data_ptr(), c.code, sa, c.pos.ptr(), c.pos.kind, c.pos.strides,
                          d.idx.mutable_data_ptr<int32_t>(), d.val.mutable_data_ptr<float>(), d.s, c.B, c.H, c.U, c.P, c.T, c.E,
                          c.Kw, c.Kr, c.rho_w, c.rho_r, 0, 1, 1, c.device.index(), stream));
    return d;
}

struct Outcome {
    Tensor y, slot, mass;
};

// prefill forward; slot / mass undefined: zero rows and mass_init.  inplace: the state tensors themselves are updated.
Outcome prefill(const Call &c, const Tensor &w, const Tensor &r, const Tensor &x, const Tensor &gamma, const Tensor &slot,
                const Tensor &mass, bool inplace, Decoded *keep) {
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(c.device.index());
    Decoded d = decode_addresses(c, w, r, stream);
    Outcome o{empty({c.B, c.T, c.H, c.C}, x.scalar_type(), c.device), inplace ? slot : empty({c.B, c.H, c.A, c.C}, at::kFloat, c.device),
              inplace ? mass : empty({c.B, c.H, c.A}, at::kFloat, c.device)};
    const int64_t bytes = rn_gsu_workspace_bytes(c.B, c.H, c.T, c.A, c.C, c.Kw, c.Kr, c.device.index());
    TORCH_CHECK(bytes >= 0, rn_last_error());
    Tensor ws = workspace(c.device, stream, bytes);
    const Rows sx(x), sg(gamma), sy(o.y);
    const int64_t sm[2] = {c.mask.defined() ? c.mask.stride(0) : 0, c.mask.defined() ? c.mask.stride(1) : 0};
    check(rn_gsu_fwd_init(d.idx.const_data_ptr<int32_t>(), d.val.const_data_ptr<float>(), d.s, x.const_data_ptr(), sx.s,
                          gamma.const_data_ptr(), sg.s, c.code, c.mask_ptr(), sm,
                          slot.defined() ? slot.const_data_ptr<float>() : nullptr, mass.defined() ? mass.const_data_ptr<float>() : nullptr,
                          c.mass_init, o.slot.mutable_data_ptr<float>(), o.mass.mutable_data_ptr<float>(), o.y.mutable_data_ptr(), sy.s,
                          ws.mutable_data_ptr(), ws.numel(), c.B, c.H, c.T, c.A, c.C, c.Kw, c.Kr, c.mass_aware, c.eps, c.device.index(),
                          stream));
    if (keep) *keep = std::move(d);
    return o;
}

// (B,T,H,C) as the backward kernels take it: channels contiguous, rows aligned to four elements
bool rows_of_four(const Tensor &t) {
    const uintptr_t align = 4 * t.element_size();
    return t.stride(3) == 1 && ((t.stride(0) | t.stride(1) | t.stride(2)) & 3) == 0 &&
           reinterpret_cast<uintptr_t>(t.const_data_ptr()) % align == 0;
}

// Prefill under autograd: one node instead of two operator nodes, an axis move per tensor and their Python formulas.
struct RamAttention : public torch::autograd::Function<RamAttention> {
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext *ctx, const Tensor &w, const Tensor &r,
                                                  const Tensor &x, const Tensor &gamma, const std::optional<Tensor> &slot_,
                                                  const std::optional<Tensor> &mass_, const Call &c) {
        const Tensor slot = slot_.value_or(Tensor()), mass = mass_.value_or(Tensor());
        Decoded d;
        Outcome o = prefill(c, w, r, x, gamma, slot, mass, false, &d);
        ctx->save_for_backward({w, r, x, gamma, slot, mass, d.idx, d.val, c.mask, c.pos.t});
        ctx->saved_data["ints"] = c10::IValue(std::vector<int64_t>{c.B, c.T, c.H, c.U, c.P, c.A, c.C, c.E, c.Kw, c.Kr, c.mass_aware,
                                                                   c.code, c.pos.kind, c.pos.strides[0], c.pos.strides[1]});
        ctx->saved_data["floats"] = c10::IValue(std::vector<double>{c.rho_w, c.rho_r, c.eps, c.mass_init});
        ctx->set_materialize_grads(false);
        return {o.y, o.slot, o.mass};
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        torch::autograd::variable_list out(7);  // w, r, x, gamma, slot, mass and the call
        Tensor dy = grads[0], dslot_post = grads[1], dmass_post = grads[2];
        if (!dy.defined() && !dslot_post.defined() && !dmass_post.defined()) return out;
        const auto saved = ctx->get_saved_variables();
        const Tensor &w = saved[0], &r = saved[1], &x = saved[2], &gamma = saved[3], &slot = saved[4], &mass = saved[5],
                     &idx = saved[6], &val = saved[7];
        const auto v = ctx->saved_data["ints"].toIntVector();
        const auto f = ctx->saved_data["floats"].toDoubleVector();
        Call c{v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], f[0], f[1], f[2], f[3], v[10] != 0, int(v[11]), x.device(), {}, {}};
        c.mask = saved[8];
        c.pos.t = saved[9];
        c.pos.kind = int(v[12]);
        c.pos.strides[0] = v[13];
        c.pos.strides[1] = v[14];
        // a call under create_graph runs with gradients enabled; the results here are constants either way, as those of
        // the registered backward operators are
        at::AutoDispatchBelowADInplaceOrView below;
        if (!dy.defined()) dy = at::zeros({c.B, c.T, c.H, c.C}, x.options());
        if (!rows_of_four(dy)) dy = dy.contiguous();
        if (dslot_post.defined()) dslot_post = dslot_post.contiguous();
        if (dmass_post.defined()) dmass_post = dmass_post.contiguous();
        const bool want_dslot = slot.defined() && ctx->needs_input_grad(4), want_dmass = mass.defined() && ctx->needs_input_grad(5);

        const int64_t K = c.Kw + c.Kr;
        Tensor dval = empty({c.B, c.T, c.H, K}, at::kFloat, c.device);
        Tensor dx = empty({c.B, c.T, c.H, c.C}, x.scalar_type(), c.device);
        Tensor dgamma = empty({c.B, c.H, c.T}, at::kFloat, c.device);
        // the state and its gradients where they exist; a state that was not given is zeros and mass_init, gradients that did not
        // come are zeros
        Tensor dslot, dmass;
        if (want_dslot) dslot = empty({c.B, c.H, c.A, c.C}, at::kFloat, c.device);
        if (want_dmass) dmass = empty({c.B, c.H, c.A}, at::kFloat, c.device);
        auto in = [](const Tensor &v) { return v.defined() ? v.const_data_ptr<float>() : nullptr; };
        const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(c.device.index());
        const int64_t bytes = rn_gsu_bwd_workspace_bytes(c.B, c.H, c.T, c.A, c.C, c.Kw, c.Kr, c.device.index());
        TORCH_CHECK(bytes >= 0, rn_last_error());
        Tensor ws = empty({std::max<int64_t>(bytes, 256)}, at::kByte, c.device);
        const int64_t sv[4] = {c.T * c.H * K, K, 1, c.H * K};
        const Rows sx(x), sg(gamma), sdy(dy), sdx(dx);
        const int64_t sm[2] = {c.mask.defined() ? c.mask.stride(0) : 0, c.mask.defined() ? c.mask.stride(1) : 0};
        check(rn_gsu_bwd_init(idx.const_data_ptr<int32_t>(), val.const_data_ptr<float>(), sv, x.const_data_ptr(), sx.s,
                              gamma.const_data_ptr(), sg.s, c.code, c.mask_ptr(), sm, in(slot), in(mass), c.mass_init, dy.const_data_ptr(),
                              sdy.s, in(dslot_post), in(dmass_post), dval.mutable_data_ptr<float>(), sv, dx.mutable_data_ptr(), sdx.s,
                              dgamma.mutable_data_ptr<float>(), want_dslot ? dslot.mutable_data_ptr<float>() : nullptr,
                              want_dmass ? dmass.mutable_data_ptr<float>() : nullptr, ws.mutable_data_ptr(), ws.numel(), c.B, c.H, c.T,
                              c.A, c.C, c.Kw, c.Kr, c.mass_aware, c.eps, c.device.index(), stream));
        if (ctx->needs_input_grad(0) || ctx->needs_input_grad(1)) {
            Tensor dw = empty({c.B, c.T, c.H, c.U, c.P}, w.scalar_type(), c.device), dr = empty({c.B, c.T, c.H, c.U, c.P}, w.scalar_type(), c.device);
            int64_t sa[5], sd[5];
            swap_axes(w, sa);
            swap_axes(dw, sd);
            check(rn_addr_bwd_pos(idx.const_data_ptr<int32_t>(), val.const_data_ptr<float>(), sv, dval.const_data_ptr<float>(), sv, w.const_data_ptr(),
                                  r.const_data_ptr(), c.code, sa, c.pos.ptr(), c.pos.kind, c.pos.strides, dw.mutable_data_ptr(),
                                  dr.mutable_data_ptr(), sd, c.B, c.H, c.U, c.P, c.T, c.E, c.Kw, c.Kr, c.rho_w, c.rho_r, 0, 1, c.device.index(),
                                  stream));
            if (ctx->needs_input_grad(0)) out[0] = dw;
            if (ctx->needs_input_grad(1)) out[1] = dr;
        }
        if (ctx->needs_input_grad(2)) out[2] = dx;
        if (ctx->needs_input_grad(3)) out[3] = dgamma.permute({0, 2, 1}).to(gamma.scalar_type());
        if (want_dslot) out[4] = dslot;
        if (want_dmass) out[5] = dmass;
        return out;
    }
};

PyObject *outcome(const Tensor &y, const Tensor &slot, const Tensor &mass) {
    PyObject *py = THPVariable_Wrap(y), *ps = THPVariable_Wrap(slot), *pm = THPVariable_Wrap(mass);
    PyObject *state = py && ps && pm ? PyTuple_Pack(2, ps, pm) : nullptr;
    PyObject *out = state ? PyTuple_Pack(2, py, state) : nullptr;
    Py_XDECREF(py);
    Py_XDECREF(ps);
    Py_XDECREF(pm);
    Py_XDECREF(state);
    return out;
}

#define RN_DECLINE_UNLESS(cond) \
    do {                        \
        if (!(cond)) Py_RETURN_NONE; \
    } while (0)

// attention(w_addr, r_addr, values, gamma, init_ram, mask, embed_num, position_ids, top_k, top_k_re_norm, mass_aware,
//           eps, t_dim, inplace, impl_backend) -> (y, (slot, mass)) or None
PyObject *attention(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 15, "attention() takes 15 arguments");
    Tensor w, r, x, gamma, slot, mass;
    RN_DECLINE_UNLESS(plain_tensor(a[0], &w) && plain_tensor(a[1], &r) && plain_tensor(a[2], &x));
    int64_t t_dim;
    RN_DECLINE_UNLESS(take_int(a[12], &t_dim) && t_dim == 1 && w.dim() == 5 && x.dim() == 4);
    Call c;
    c.B = w.size(0); c.T = w.size(1); c.H = w.size(2); c.U = w.size(3); c.P = w.size(4); c.C = x.size(3);
    c.device = w.device();
    c.code = dtype_code(w.scalar_type());
    RN_DECLINE_UNLESS(c.code >= 0 && r.scalar_type() == w.scalar_type() && x.scalar_type() == w.scalar_type());
    RN_DECLINE_UNLESS(r.sizes() == w.sizes() && x.size(0) == c.B && x.size(1) == c.T && x.size(2) == c.H);
    RN_DECLINE_UNLESS(r.device() == c.device && x.device() == c.device && w.numel() > 0 && x.numel() > 0);
    c.A = 1;
    for (int64_t u = 0; u < c.U; ++u) {
        c.A *= c.P;
        RN_DECLINE_UNLESS(c.A < (int64_t(1) << 30));
    }
    const bool gate_tensor = plain_tensor(a[3], &gamma);
    double gate_value = 0.0;
    if (gate_tensor) RN_DECLINE_UNLESS(gamma.dim() == 3 && gamma.size(0) == c.B && gamma.size(1) == c.T && gamma.size(2) == c.H &&
                                       gamma.scalar_type() == w.scalar_type() && gamma.device() == c.device);
    else RN_DECLINE_UNLESS(take_float(a[3], &gate_value));

    c.mass_init = 1.0 / double(c.A);
    if (a[4] != Py_None) {
        RN_DECLINE_UNLESS(PyTuple_Check(a[4]) && PyTuple_GET_SIZE(a[4]) == 2);
        RN_DECLINE_UNLESS(plain_tensor(PyTuple_GET_ITEM(a[4], 0), &slot) && plain_tensor(PyTuple_GET_ITEM(a[4], 1), &mass));
        RN_DECLINE_UNLESS(slot.dim() == 4 && slot.size(0) == c.B && slot.size(1) == c.H && slot.size(2) == c.A && slot.size(3) == c.C);
        RN_DECLINE_UNLESS(mass.dim() == 3 && mass.size(0) == c.B && mass.size(1) == c.H && mass.size(2) == c.A);
        RN_DECLINE_UNLESS(slot.scalar_type() == at::kFloat && mass.scalar_type() == at::kFloat && slot.is_contiguous() && mass.is_contiguous());
        RN_DECLINE_UNLESS(slot.device() == c.device && mass.device() == c.device);
        RN_DECLINE_UNLESS(reinterpret_cast<uintptr_t>(slot.const_data_ptr()) % 16 == 0);
    }
    if (a[5] != Py_None) {
        RN_DECLINE_UNLESS(plain_tensor(a[5], &c.mask) && c.mask.scalar_type() == at::kBool && c.mask.device() == c.device);
        RN_DECLINE_UNLESS(c.mask.dim() == 2 && c.mask.size(0) == c.B && c.mask.size(1) == c.T);
    }
    RN_DECLINE_UNLESS(take_int(a[6], &c.E) && c.E >= 0 && c.E <= c.H);
    RN_DECLINE_UNLESS(take_positions(a[7], c.B, c.T, c.device, &c.pos));
    RN_DECLINE_UNLESS(take_pair(a[8], &c.Kw, &c.Kr, take_int));
    RN_DECLINE_UNLESS(c.Kw > 0 && c.Kr > 0 && c.Kw <= c.A && c.Kr <= c.A && c.Kw <= 128 && c.Kr <= 128);
    RN_DECLINE_UNLESS(take_pair(a[9], &c.rho_w, &c.rho_r, take_float));
    RN_DECLINE_UNLESS(c.rho_w >= 0 && c.rho_w <= 1 && c.rho_r >= 0 && c.rho_r <= 1);
    RN_DECLINE_UNLESS(PyBool_Check(a[10]) && PyBool_Check(a[13]));
    c.mass_aware = a[10] == Py_True;
    const bool inplace = a[13] == Py_True;
    RN_DECLINE_UNLESS(take_float(a[11], &c.eps) && c.eps > 0);
    RN_DECLINE_UNLESS(a[14] == Py_None || (PyUnicode_Check(a[14]) && PyUnicode_CompareWithASCIIString(a[14], "cuda") == 0));
    RN_DECLINE_UNLESS(!inplace || slot.defined());
    // int32 slot numbers and event counts, T counted in whole 32s as the front end does
    const int64_t T32 = (c.T + 31) / 32 * 32;
    RN_DECLINE_UNLESS(c.U <= 8 && c.P <= 128 && c.B * c.H * c.A < INT_LIMIT && c.B * c.H * T32 * (c.Kw + c.Kr) < INT_LIMIT);
    RN_DECLINE_UNLESS(plain_context());

    const bool differentiable = w.requires_grad() || r.requires_grad() || x.requires_grad() || (gate_tensor && gamma.requires_grad()) ||
                                (slot.defined() && (slot.requires_grad() || mass.requires_grad()));
    RN_DECLINE_UNLESS(!(inplace && differentiable));
    if (!gate_tensor) gamma = at::full({c.B, c.T, c.H}, gate_value, x.options());

    if (c.T == 1 && !differentiable) {
        int64_t ld[5];
        RN_DECLINE_UNLESS(c.C <= 1024 && contiguous_rows(w, &ld[0]) && contiguous_rows(r, &ld[1]) && contiguous_rows(x, &ld[2]) &&
                          contiguous_rows(gamma, &ld[3]));
        RN_DECLINE_UNLESS(!c.mask.defined() || c.B == 1 || c.mask.stride(0) == 1);
        ld[4] = c.H * c.C;
        RECORD_FUNCTION("ramnet_ops::decode_step", std::vector<c10::IValue>());
        if (!slot.defined()) {
            slot = at::zeros({c.B, c.H, c.A, c.C}, x.options().dtype(at::kFloat));
            mass = at::full({c.B, c.H, c.A}, c.mass_init, x.options().dtype(at::kFloat));
        } else if (!inplace) {
            slot = slot.clone();
            mass = mass.clone();
        }
        Tensor y = empty({c.B, 1, c.H, c.C}, x.scalar_type(), c.device);
        check(rn_decode_step_pos(w.const_data_ptr(), r.const_data_ptr(), x.const_data_ptr(), gamma.const_data_ptr(), c.code,
                                 slot.mutable_data_ptr<float>(), mass.mutable_data_ptr<float>(), c.mask_ptr(), c.pos.ptr(), c.pos.kind,
                                 c.pos.strides[0], y.mutable_data_ptr(), nullptr, nullptr, 0.0, nullptr, nullptr, ld, c.B, c.H, c.U, c.P, c.C,
                                 c.E, c.Kw, c.Kr, c.rho_w, c.rho_r, c.mass_aware, c.eps, c.device.index(),
                                 c10::cuda::getCurrentCUDAStream(c.device.index())));
        return outcome(y, slot, mass);
    }
    RN_DECLINE_UNLESS(r.strides() == w.strides() && x.stride(3) == 1);
    if (differentiable && at::GradMode::is_enabled()) {
        RN_DECLINE_UNLESS(c.C % 4 == 0 && rows_of_four(x));
        const auto some = [](const Tensor &t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
        const auto out = RamAttention::apply(w, r, x, gamma, some(slot), some(mass), c);
        return outcome(out[0], out[1], out[2]);
    }
    RECORD_FUNCTION("ramnet_ops::prefill", std::vector<c10::IValue>());
    const Outcome o = prefill(c, w, r, x, gamma, slot, mass, inplace, nullptr);
    return outcome(o.y, o.slot, o.mass);
    END_HANDLE_TH_ERRORS
}

// topk_addr(addr, embed_num, position_ids, top_k, top_k_re_norm, addr_val_neg, encode_batch_idx) -> (idx, val) or None
PyObject *topk_addr(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 7, "topk_addr() takes 7 arguments");
    Tensor addr;
    RN_DECLINE_UNLESS(plain_tensor(a[0], &addr) && addr.dim() == 5 && addr.numel() > 0);
    const int64_t B = addr.size(0), H = addr.size(1), U = addr.size(2), P = addr.size(3), T = addr.size(4);
    const int code = dtype_code(addr.scalar_type());
    RN_DECLINE_UNLESS(code >= 0 && U <= 8 && P <= 128 && !(addr.requires_grad() && at::GradMode::is_enabled()));
    int64_t A = 1, E, K;
    for (int64_t u = 0; u < U; ++u) A *= P;
    double rho;
    Positions pos;
    RN_DECLINE_UNLESS(take_int(a[1], &E) && E >= 0 && E <= H);
    RN_DECLINE_UNLESS(a[2] != Py_None && take_positions(a[2], B, T, addr.device(), &pos) && pos.t.size(0) == B);
    RN_DECLINE_UNLESS(take_int(a[3], &K) && K > 0 && K <= A && K <= 128 && take_float(a[4], &rho) && rho >= 0 && rho <= 1);
    RN_DECLINE_UNLESS(PyBool_Check(a[5]) && PyBool_Check(a[6]));
    const int64_t T32 = (T + 31) / 32 * 32;
    RN_DECLINE_UNLESS(A < (int64_t(1) << 30) && B * H * A < INT_LIMIT && B * H * K * T32 < INT_LIMIT && B * H * U * P * T32 < INT_LIMIT);
    RN_DECLINE_UNLESS(plain_context());
    RECORD_FUNCTION("ramnet_ops::topk_addr", std::vector<c10::IValue>());
    const at::Device device = addr.device();
    Tensor idx = empty({B, T, H, K}, at::kInt, device), val = empty({B, T, H, K}, at::kFloat, device);
    const int64_t sa[5] = {addr.stride(0), addr.stride(1), addr.stride(2), addr.stride(3), addr.stride(4)}, so[4] = {T * H * K, K, 1, H * K};
    check(rn_addr_fwd_pos(addr.const_data_ptr(), nullptr, code, sa, pos.ptr(), pos.kind, pos.strides, idx.mutable_data_ptr<int32_t>(),
                          val.mutable_data_ptr<float>(), so, B, H, U, P, T, E, K, 0, rho, 0.0, a[5] == Py_True, 0, a[6] == Py_True, device.index(),
                          c10::cuda::getCurrentCUDAStream(device.index())));
    PyObject *pi = THPVariable_Wrap(idx.permute({0, 2, 3, 1})), *pv = THPVariable_Wrap(val.permute({0, 2, 3, 1}));
    PyObject *out = pi && pv ? PyTuple_Pack(2, pi, pv) : nullptr;
    Py_XDECREF(pi);
    Py_XDECREF(pv);
    return out;
    END_HANDLE_TH_ERRORS
}

// workspace(device_index, stream, bytes) -> uint8 tensor
PyObject *py_workspace(PyObject *, PyObject *args) {
    HANDLE_TH_ERRORS
    int device;
    unsigned long long stream;
    long long bytes;
    if (!PyArg_ParseTuple(args, "iKL", &device, &stream, &bytes)) return nullptr;
    return THPVariable_Wrap(workspace(at::Device(at::kCUDA, c10::DeviceIndex(device)), reinterpret_cast<cudaStream_t>(stream), bytes));
    END_HANDLE_TH_ERRORS
}

PyObject *py_release(PyObject *, PyObject *) {
    HANDLE_TH_ERRORS
    std::map<std::pair<int, cudaStream_t>, Tensor> gone;
    {
        std::lock_guard<std::mutex> lock(g_ws_lock);
        gone.swap(ws_table());
    }
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(attention)), METH_FASTCALL, nullptr},
    {"topk_addr", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(topk_addr)), METH_FASTCALL, nullptr},
    {"workspace", py_workspace, METH_VARARGS, nullptr},
    {"release_workspaces", py_release, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
