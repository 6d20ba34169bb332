// The autograd side of the scans in C++: what scan(), scan_single() and scan_gated() do for ordinary
// calls (plain CUDA tensors, no autocast, no function transform), without Python frames in the forward
// or in the autograd engine's thread.  Each entry returns None for a call it does not take; the caller
// then goes the Python way, which also words all refusals.
//
// What bounds small calls is host time: a training step of B2 T1024 D768 runs 17 us of kernels.  Its
// two launches through Python classes took 129 us a step, through these 76; decoding 33 and 13 us a call.
//
// The library is reached through the addresses that the package's ctypes table holds, and the streams'
// workspaces stay with workspace.py: one Python call per launch takes the device's lock and returns what
// the context is made of.  The GIL is held for such calls only, not for allocations, copies and launches,
// any of which may block (memory to reclaim, a full launch queue).
#include <torch/extension.h>

#include "../../include/fss_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Library {
    decltype(&fss_scan_forward_ex) forward;
    decltype(&fss_scan_backward_ex) backward;
    decltype(&fss_scan_forward_gated) forward_gated;
    decltype(&fss_scan_backward_gated) backward_gated;
} lib;
// Python: acquire(device index, B, T, D, dtype id, gated backward) -> (context, its address, release of the
// device's lock, workspace or None); launched(workspace); check(code, where); the gated backward for any
// layout.  Held for the process's life.
PyObject *py_acquire, *py_launched, *py_check, *py_gated_backward;

struct Shape {
    int64_t B, T, D;
    int dtype;
    explicit Shape(const Tensor &t) : B(t.size(0)), T(t.size(1)), D(t.size(2)), dtype(t.scalar_type() == at::kBFloat16 ? FSS_DTYPE_BF16 : FSS_DTYPE_F32) {}
};

// One launch, with a context of its own, made without the GIL.  The device's lock (workspace.py) is held
// from the look-up of the workspace until the launch is recorded, by the thread that makes the launch.
struct Launch {
    fss_scan_ctx ctx;
    PyObject *release = nullptr, *workspace = nullptr;      // owned; None: nobody wants to hear of the launch
    Launch(const Tensor &t, const Shape &s, int flags, bool gated_backward = false) {
        py::gil_scoped_acquire gil;
        const py::object got = py::reinterpret_steal<py::object>(PyObject_CallFunction(py_acquire, "iLLLii", (int)t.get_device(), (long long)s.B,
                                                                                       (long long)s.T, (long long)s.D, s.dtype, (int)gated_backward));
        if (!got) throw py::error_already_set();
        const auto item = [&](int k) { return PyTuple_GET_ITEM(got.ptr(), k); };
        ctx = *reinterpret_cast<const fss_scan_ctx *>(PyLong_AsUnsignedLongLong(item(1)));      // (item 0 keeps it alive)
        ctx.flags |= flags;
        release = Py_NewRef(item(2));
        workspace = Py_NewRef(item(3));
    }
    Launch(const Launch &) = delete;
    ~Launch() {
        if (!release) return;
        py::gil_scoped_acquire gil;
        py::error_scope keep;      // (an error that is on its way)
        give_back();
        PyErr_Clear();
    }
    // after the call of the library
    void done(int rc = FSS_OK, const char *where = nullptr) {
        py::gil_scoped_acquire gil;
        if (workspace != Py_None) py::reinterpret_borrow<py::object>(py_launched)(py::handle(workspace));
        give_back();
        if (rc != FSS_OK) py::reinterpret_borrow<py::object>(py_check)(rc, where);      // raises
    }

  private:
    void give_back() {
        Py_XDECREF(PyObject_CallNoArgs(release));
        Py_CLEAR(release);
        Py_CLEAR(workspace);
    }
};

// unit channel stride, rows and batches that do not overlap
Tensor rowwise(const Tensor &t) {
    if (t.is_contiguous()) return t;
    const int64_t B = t.size(0), T = t.size(1), D = t.size(2);
    const bool ok = (D == 1 || t.stride(2) == 1) && (T == 1 || t.stride(1) >= D) && (B == 1 || t.stride(0) >= (T - 1) * t.stride(1) + D);
    return ok ? t : t.contiguous();
}
fss_view view(const Tensor &t) {
    const int64_t B = t.size(0), T = t.size(1), D = t.size(2);
    if (t.is_contiguous()) return {t.data_ptr(), std::max<int64_t>(T * D, 1), D};
    const int64_t st = T > 1 ? t.stride(1) : D;
    return {t.data_ptr(), B > 1 ? t.stride(0) : std::max<int64_t>(st * T, 1), st};
}
// what the single-pass kernels can address
bool addressable(const Tensor &t) {
    const int64_t per16 = 16 / t.element_size();
    if (t.size(2) % per16 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 || (t.size(2) > 1 && t.stride(2) != 1)) return false;
    return !((t.size(1) > 1 && t.stride(1) % per16) || (t.size(0) > 1 && t.stride(0) % per16));
}
Tensor placed(const Tensor &t) {      // a copy where only the placement, not the width, is in the way
    if (t.size(2) % (16 / t.element_size()) || addressable(t)) return t;
    return t.clone(at::MemoryFormat::Contiguous);
}
Tensor like(const Tensor &t) { return at::empty(t.sizes(), t.options().memory_format(at::MemoryFormat::Contiguous)); }

bool ordinary(const Tensor &t, const Tensor &first, at::ScalarType dtype) {
    return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.scalar_type() == dtype && t.dim() == 3 &&
           t.sizes() == first.sizes() && t.device() == first.device() && t.numel() > 0;
}
bool ordinary_vector(const Tensor &t, const Tensor &like, at::IntArrayRef sizes) {
    return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.scalar_type() == at::kFloat && t.device() == like.device() &&
           t.sizes() == sizes && t.is_contiguous();
}
// What the backward unpacks need not be what the forward saved: saved-tensor hooks may return anything.
// The engine has checked the gradients against the outputs, so the saved tensors are checked against them.
void check_unpacked(const Tensor &t, const Tensor &grad, const char *name) {
    TORCH_CHECK(ordinary(t, grad, grad.scalar_type()), name, ": the saved tensor came back as ", t.toString(), t.sizes(), " on ", t.device(),
                ", expected ", grad.toString(), grad.sizes(), " on ", grad.device());
}

struct Scan : torch::autograd::Function<Scan> {
    static variable_list forward(AutogradContext *ctx, const Tensor &alpha, const Tensor &beta, const std::optional<Tensor> &state0, bool want_final,
                                 bool reverse) {
        const Shape s(alpha);
        const Tensor h0 = state0 ? *state0 : Tensor();
        const Tensor a = rowwise(alpha), b = rowwise(beta), h = like(alpha);
        Tensor last;
        if (want_final) last = at::empty({s.B, s.D}, alpha.options().dtype(at::kFloat));
        fss_forward_state state{};
        state.h_in = h0.defined() ? h0.data_ptr<float>() : nullptr;
        state.h_last = last.defined() ? last.data_ptr<float>() : nullptr;
        const fss_view va = view(a), vb = view(b), vh = view(h);
        Launch go(alpha, s, (h0.defined() ? FSS_FLAG_CONTINUATION : 0) | (reverse ? FSS_FLAG_REVERSE : 0));
        go.done(lib.forward(&go.ctx, s.dtype, s.B, s.T, s.D, &va, &vb, &vh, h0.defined() || want_final ? &state : nullptr),
                "fss_scan_forward_ex");
        ctx->save_for_backward({alpha, h, h0});
        ctx->saved_data["reverse"] = reverse;
        if (want_final) return {h, last};
        return {h};
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list saved = ctx->get_saved_variables();
        const Tensor &alpha = saved[0], &h0 = saved[2];
        check_unpacked(alpha, grads[0], "alpha_saved");
        check_unpacked(saved[1], grads[0], "h_saved");
        TORCH_CHECK(!h0.defined() || ordinary_vector(h0, alpha, {alpha.size(0), alpha.size(2)}),
                    "h_prev: expected a contiguous fp32 CUDA tensor of ", alpha.size(0), "x", alpha.size(2), " elements");
        const bool reverse = ctx->saved_data["reverse"].toBool();
        const Shape s(alpha);
        const Tensor a = rowwise(alpha), h = rowwise(saved[1]);
        Tensor g = rowwise(grads[0]);
        if (reverse) g = placed(g);
        Tensor u_in, u_out;
        if (grads.size() > 1 && grads[1].defined()) u_in = grads[1].to(at::kFloat).contiguous();
        if (h0.defined()) u_out = at::empty({s.B, s.D}, alpha.options().dtype(at::kFloat));
        const Tensor da = like(alpha), db = like(alpha);
        fss_backward_state state{};
        state.u_in = u_in.defined() ? u_in.data_ptr<float>() : nullptr;
        state.h_prev = h0.defined() ? h0.data_ptr<float>() : nullptr;
        state.u_out = u_out.defined() ? u_out.data_ptr<float>() : nullptr;
        const fss_view va = view(a), vh = view(h), vg = view(g), vda = view(da), vdb = view(db);
        Launch go(alpha, s, (h0.defined() ? FSS_FLAG_CONTINUATION : 0) | (reverse ? FSS_FLAG_REVERSE : 0));
        go.done(lib.backward(&go.ctx, s.dtype, s.B, s.T, s.D, &va, &vh, &vg, &vda, &vdb, u_in.defined() || h0.defined() ? &state : nullptr),
                "fss_scan_backward_ex");
        return {da, db, u_out, Tensor(), Tensor()};
    }
};

struct Gated : torch::autograd::Function<Gated> {
    static Tensor forward(AutogradContext *ctx, const Tensor &r, const Tensor &i, const Tensor &x, const Tensor &lam) {
        const Shape s(r);
        const Tensor h = like(r);
        const fss_view vr = view(r), vi = view(i), vx = view(x), vh = view(h);
        Launch go(r, s, 0);
        go.done(lib.forward_gated(&go.ctx, s.dtype, s.B, s.T, s.D, &vr, &vi, &vx, lam.data_ptr<float>(), &vh, nullptr),
                "fss_scan_forward_gated");
        ctx->save_for_backward({r, i, x, lam, h});
        return h;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list saved = ctx->get_saved_variables();
        const Tensor &r = saved[0], &lam = saved[3];
        const auto any_layout = [&] {      // or a refusal, worded there
            py::gil_scoped_acquire gil;
            const py::tuple out = py::reinterpret_borrow<py::object>(py_gated_backward)(r, saved[1], saved[2], lam, saved[4], grads[0]);
            return variable_list{out[0].cast<Tensor>(), out[1].cast<Tensor>(), out[2].cast<Tensor>(), out[3].cast<Tensor>()};
        };
        for (int k : {0, 1, 2, 4})
            if (!ordinary(saved[k], grads[0], grads[0].scalar_type())) return any_layout();
        if (!ordinary_vector(lam, r, {r.size(2)})) return any_layout();
        const Shape s(r);
        const Tensor g = placed(grads[0].contiguous()), dr = like(r), di = like(r), dx = like(r), dlam = at::empty_like(lam);
        const Tensor rr = rowwise(r), ri = rowwise(saved[1]), rx = rowwise(saved[2]), rh = rowwise(saved[4]);
        const fss_view vr = view(rr), vi = view(ri), vx = view(rx), vh = view(rh), vg = view(g), v0 = view(dr), v1 = view(di), v2 = view(dx);
        Launch go(r, s, 0, true);
        const int rc = lib.backward_gated(&go.ctx, s.dtype, s.B, s.T, s.D, &vr, &vi, &vx, lam.data_ptr<float>(), &vh, &vg, &v0, &v1, &v2,
                                          dlam.data_ptr<float>());
        go.done(rc == FSS_E_LAYOUT ? FSS_OK : rc, "fss_scan_backward_gated");
        if (rc == FSS_E_LAYOUT) return any_layout();      // saved-tensor hooks handed back copies that lie otherwise, say
        return {dr, di, dx, dlam};
    }
};

// alpha, beta, h0 (or None), return the final state, reverse, bf16
py::object scan(const Tensor &alpha, const Tensor &beta, const std::optional<Tensor> &h0, bool want_final, bool reverse, bool bf16) {
    const at::ScalarType dtype = bf16 ? at::kBFloat16 : at::kFloat;
    if (alpha.dim() != 3 || !ordinary(alpha, alpha, dtype) || !ordinary(beta, alpha, dtype)) return py::none();
    if (h0 && !ordinary_vector(*h0, alpha, {alpha.size(0), alpha.size(2)})) return py::none();
    if (reverse && !(addressable(alpha) && addressable(beta))) return py::none();
    const variable_list out = [&] {
        py::gil_scoped_release no_gil;
        return Scan::apply(alpha, beta, h0, want_final, reverse);
    }();
    if (want_final) return py::make_tuple(out[0], out[1]);
    return py::cast(out[0]);
}

py::object gated(const Tensor &r, const Tensor &i, const Tensor &x, const Tensor &lam) {
    if (r.dim() != 3 || (r.scalar_type() != at::kBFloat16 && r.scalar_type() != at::kFloat)) return py::none();
    for (const Tensor *t : {&r, &i, &x})
        if (!ordinary(*t, r, r.scalar_type()) || !t->is_contiguous() || !addressable(*t)) return py::none();
    if (!ordinary_vector(lam, r, {r.size(2)})) return py::none();
    const Tensor h = [&] {
        py::gil_scoped_release no_gil;
        return Gated::apply(r, i, x, lam);
    }();
    return py::cast(h);
}

void bind(uintptr_t forward, uintptr_t backward, uintptr_t forward_gated, uintptr_t backward_gated, py::object acquire, py::object launched,
          py::object check, py::object gated_backward) {
    lib.forward = reinterpret_cast<decltype(lib.forward)>(forward);
    lib.backward = reinterpret_cast<decltype(lib.backward)>(backward);
    lib.forward_gated = reinterpret_cast<decltype(lib.forward_gated)>(forward_gated);
    lib.backward_gated = reinterpret_cast<decltype(lib.backward_gated)>(backward_gated);
    py_acquire = acquire.release().ptr();
    py_launched = launched.release().ptr();
    py_check = check.release().ptr();
    py_gated_backward = gated_backward.release().ptr();
}

}  // namespace

PYBIND11_MODULE(_fss_torch, m) {
    m.def("bind", &bind);
    m.def("scan", &scan);
    m.def("gated", &gated);
}
