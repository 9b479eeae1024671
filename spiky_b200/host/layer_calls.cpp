// Host side of a layer call in native code: what the layers' forward and their autograd node do on every call - checks,
// allocations, launches - for the ordinary cases.  The launches themselves are the C-ABI library's (include/spiky_b200.h).
//
// `apply(x, layer)` returns the layer's output, or None for a call it leaves to the Python route of lut_layer.py, which
// stays the definition of every case: fixed-point layers, replaced methods and hooks, tensor subclasses, tracing and
// torch's modes, functorch transforms, forward-mode differentiation, whatever a check refuses.  Nothing is kept from one call
// for the next: every attribute is read from the layer each time.  The node's backward pass looks again, and calls the
// layer's Python method where it finds anything out of the ordinary.  It does not own the layer, which may own its output: see
// LayerNode.
//
// Measured, host time of forward and backward (Python route / this one): fully connected layer of 256 samples 231 / 110 us (59 of
// them are autograd's own for an empty function), projection layer 206 / 105, concatenation-mode layer 238 / 109; the logits of
// a four-layer transformer 607 / 314.
#include <torch/extension.h>
#include <torch/version.h>

#include <ATen/FuncTorchTLS.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_cpp_function.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "../../include/spiky_b200.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct Library {
    decltype(&lutb_nonseq_fc_forward) fc_forward;
    decltype(&lutb_nonseq_fc_backward) fc_backward;
    decltype(&lutb_nonseq_fc_backward_workspace) fc_backward_workspace;
    decltype(&lutb_nonseq_sparse_forward) sparse_forward;
    decltype(&lutb_nonseq_sparse_backward) sparse_backward;
    decltype(&lutb_concat_forward) concat_forward;
    decltype(&lutb_concat_backward) concat_backward;
    decltype(&lutb_product_forward) product_forward;
    decltype(&lutb_product_backward) product_backward;
    decltype(&lutb_product_workspace) product_workspace;
    decltype(&lutb_product_keeps_histogram) product_keeps_histogram;
    decltype(&lutb_zero_buffers) zero_buffers;
    decltype(&lutb_nonseq_fc_table_grad_rows) rows;
    decltype(&lutb_nonseq_fc_table_grad_rows_workspace) rows_workspace;
    decltype(&lutb_dense_to_sparse_workspace) cells_workspace;
    decltype(&lutb_row_cells_count) cells_count;
    decltype(&lutb_row_cells_scatter) cells_scatter;
};
Library lib;

// ------------------------------------------------------------------------------------------------ Python objects
struct Names {
    PyObject *dict_parameters, *dict_buffers, *weights, *anchors, *positional, *training, *dm, *shared_context, *cmp_eps, *device, *policy,
        *type, *normalized, *sequence_length, *concatenation, *sliced, *positional_dim, *unified, *fully_connected, *dw_variant,
        *product_variant, *sparse_rows_direct, *dm_device, *dm_fully_connected, *dm_sparse, *dm_seq_len, *dm_forward_seen, *dm_kept, *n_weights,
        *rows_per_detector, *cfg, *c_struct, *input_shape, *output_shape, *prepare_positional, *external_lr, *scratch_limit, *keep_limit;
};
Names names;
PyObject *manager_class, *manager_base, *tensor_class, *parameter_class, *policy_dense, *policy_internal, *policy_sparse, *check_status, *layer_class;
// methods whose replacement, on an instance or by a subclass, sends a call to the Python route
std::vector<std::pair<PyObject *, PyObject *>> layer_methods, manager_methods;   // (name, original)
std::vector<PyObject *> layer_hooks;
std::vector<PyObject *> layer_parts;   // names of what a layer's backward pass reads

struct Ref {   // owned reference
    PyObject *p = nullptr;
    explicit Ref(PyObject *q = nullptr) : p(q) {}
    Ref(const Ref &) = delete;
    Ref &operator=(const Ref &) = delete;
    ~Ref() { Py_XDECREF(p); }
    PyObject *get() const { return p; }
    explicit operator bool() const { return p != nullptr; }
};

PyObject *instance_dict(PyObject *o) {   // borrowed
    PyObject **d = _PyObject_GetDictPtr(o);
    return d ? *d : nullptr;
}
PyObject *item(PyObject *dict, PyObject *name) { return PyDict_GetItemWithError(dict, name); }   // borrowed
bool is_true(PyObject *o) { return o == Py_True; }
bool as_int(PyObject *o, int64_t &v) {
    if (o == nullptr || !PyLong_Check(o)) return false;
    v = PyLong_AsLongLong(o);
    return !(v == -1 && PyErr_Occurred());
}
// the object's dictionary holds none of the methods, and its class has the originals
bool methods_untouched(PyObject *o, PyObject *dict, const std::vector<std::pair<PyObject *, PyObject *>> &methods) {
    for (const auto &m : methods)
        if (item(dict, m.first) != nullptr || _PyType_Lookup(Py_TYPE(o), m.first) != m.second) return false;
    return true;
}
bool exact_tensor(PyObject *o) {
    return o != nullptr && ((PyObject *)Py_TYPE(o) == tensor_class || (PyObject *)Py_TYPE(o) == parameter_class);
}
[[noreturn]] void raise_current() {
    python_error e;
    e.persist();
    throw std::move(e);
}
void check(int status) {
    if (status == 0) return;
    Ref r(PyObject_CallFunction(check_status, "i", status));   // raises what the Python route raises
    raise_current();
}

// ------------------------------------------------------------------------------------------------ what a call needs
bool plain_cuda(const Tensor &t, at::ScalarType type, c10::DeviceIndex device) {
    if (!t.defined() || t.layout() != at::kStrided || t.scalar_type() != type || !t.is_cuda() || t.device().index() != device) return false;
    const auto keys = t.unsafeGetTensorImpl()->key_set();
    return !keys.has_any(c10::python_ks) && !keys.has(c10::DispatchKey::FuncTorchGradWrapper) && !keys.has(c10::DispatchKey::FuncTorchBatched) &&
           !keys.has(c10::DispatchKey::Functionalize) && !keys.has(c10::DispatchKey::Batched) && !t.is_neg() && !t.is_conj() && !t._is_zerotensor();
}
bool ordinary_context() {
    return !torch::jit::tracer::isTracing() && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() &&
           (at::functorch::functorchTLSAccessor() == nullptr ||   // (it stays after the first transform; a key is there while one is active)
            !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode));
}

enum Mode { NONSEQ, CONCAT, PRODUCT };

struct Call {
    PyObject *layer, *dict, *dm, *dm_dict;
    Mode mode;
    bool training, fully_connected;
    c10::DeviceIndex device;
    int64_t S, npe;
    Tensor weights, anchors;
    lutb_layer_cfg cfg;
    lutb_sparse_index sparse;
    PyObject *policy_type;
    bool normalized;
};

template <class T>
bool copy_struct(PyObject *o, T &out) {
    Py_buffer b;
    if (o == nullptr || PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) return false;
    const bool ok = b.len == (Py_ssize_t)sizeof(T);
    if (ok) std::memcpy(&out, b.buf, sizeof(T));
    PyBuffer_Release(&b);
    return ok;
}

// False: not a call for this route.  (The caller clears what a failed look-up may have raised.)
bool read_layer(PyObject *layer, Call &c, bool backward) {
    c.layer = layer;
    c.dict = instance_dict(layer);
    if (c.dict == nullptr || !methods_untouched(layer, c.dict, layer_methods)) return false;
    for (PyObject *h : layer_hooks) {
        PyObject *v = item(c.dict, h);
        if ((v != nullptr && v != Py_None) || _PyType_Lookup(Py_TYPE(layer), h) != nullptr) return false;
    }
    c.dm = item(c.dict, names.dm);
    if (c.dm == nullptr || (PyObject *)Py_TYPE(c.dm) != manager_class) return false;   // (fixed-point layers: Python)
    c.dm_dict = instance_dict(c.dm);
    if (c.dm_dict == nullptr || !methods_untouched(c.dm, c.dm_dict, manager_methods)) return false;
    int64_t device, S;
    if (!as_int(item(c.dm_dict, names.dm_device), device) || device < 0 || !as_int(item(c.dict, names.sequence_length), S)) return false;
    c.device = (c10::DeviceIndex)device;
    PyObject *dev = item(c.dict, names.device);
    if (dev == nullptr || !THPDevice_Check(dev)) return false;
    const at::Device own = reinterpret_cast<THPDevice *>(dev)->device;
    if (!own.is_cuda() || own.index() != c.device) return false;
    c.S = S;
    PyObject *concat = item(c.dict, names.concatenation);
    c.mode = S == 1 ? NONSEQ : is_true(concat) ? CONCAT : PRODUCT;
    PyObject *npe = item(c.dict, names.positional_dim);
    c.npe = 0;
    if (npe != nullptr && npe != Py_None && !as_int(npe, c.npe)) return false;
    PyObject *training = item(c.dict, names.training);
    if (training != Py_True && training != Py_False) return false;
    c.training = is_true(training);
    PyObject *fc = item(c.dm_dict, names.dm_fully_connected);
    if (fc != Py_True && fc != Py_False) return false;
    c.fully_connected = is_true(fc);
    if (is_true(item(c.dict, names.fully_connected)) != c.fully_connected) return false;
    if (c.mode != NONSEQ && !c.fully_connected) return false;
    int64_t dm_seq;
    if (!as_int(item(c.dm_dict, names.dm_seq_len), dm_seq) || dm_seq != (c.mode == CONCAT ? S : 1)) return false;

    PyObject *params = item(c.dict, names.dict_parameters), *buffers = item(c.dict, names.dict_buffers);
    if (params == nullptr || buffers == nullptr) return false;
    PyObject *w = item(params, names.weights), *a = item(buffers, names.anchors);
    if (!exact_tensor(w) || !exact_tensor(a)) return false;
    c.weights = THPVariable_Unpack(w);
    c.anchors = THPVariable_Unpack(a);
    if (!plain_cuda(c.weights, at::kFloat, c.device) || !plain_cuda(c.anchors, at::kInt, c.device)) return false;
    if (c.weights.dim() != 1 || c.anchors.dim() != 1 || !c.weights.is_contiguous() || !c.anchors.is_contiguous()) return false;

    PyObject *policy = item(c.dict, names.policy), *policy_dict = policy ? instance_dict(policy) : nullptr;
    if (policy_dict == nullptr) return false;
    c.policy_type = item(policy_dict, names.type);
    c.normalized = is_true(item(policy_dict, names.normalized));

    // the dead band counts in the forward pass, and in both of product mode
    PyObject *context = item(c.dict, names.shared_context), *context_dict = context ? instance_dict(context) : nullptr;
    PyObject *eps = context_dict ? item(context_dict, names.cmp_eps) : nullptr;
    if (eps == nullptr || !(PyFloat_Check(eps) || PyLong_Check(eps))) return false;
    const bool with_eps = !backward || c.mode == PRODUCT;
    Ref zero(PyFloat_FromDouble(0.0));
    PyObject *sliced = c.mode == PRODUCT ? item(c.dict, names.sliced) : Py_False;
    if (sliced == nullptr) return false;
    Ref cfg(PyObject_CallMethodObjArgs(c.dm, names.cfg, with_eps ? eps : zero.get(), sliced, nullptr));
    if (!cfg || !copy_struct(cfg.get(), c.cfg)) {
        PyErr_Clear();
        return false;
    }
    int64_t n_weights;
    if (c.fully_connected) {
        int64_t rows;
        if (!as_int(item(c.dm_dict, names.rows_per_detector), rows)) return false;
        n_weights = rows * c.cfg.n_detectors * c.cfg.n_outputs;
    } else {
        PyObject *index = item(c.dm_dict, names.dm_sparse);
        if (index == nullptr || index == Py_None) return false;
        Ref n(PyObject_GetAttr(index, names.n_weights)), s(PyObject_CallMethodNoArgs(index, names.c_struct));
        if (!n || !s || !as_int(n.get(), n_weights) || !copy_struct(s.get(), c.sparse)) {
            PyErr_Clear();
            return false;
        }
    }
    return c.weights.numel() == n_weights && c.anchors.numel() == (int64_t)c.cfg.n_detectors * c.cfg.n_anchors * 2;
}

// Appends the layer's own shape (a tuple of ints); false when it is something else.
bool append_shape(PyObject *layer, PyObject *method, std::vector<int64_t> &out) {
    Ref t(PyObject_CallMethodNoArgs(layer, method));
    if (!t || !PyTuple_Check(t.get())) {
        PyErr_Clear();
        return false;
    }
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(t.get()); i++) {
        int64_t v;
        if (!as_int(PyTuple_GET_ITEM(t.get(), i), v)) {
            PyErr_Clear();
            return false;
        }
        out.push_back(v);
    }
    return true;
}

float *f32(const Tensor &t) { return t.defined() ? static_cast<float *>(t.data_ptr()) : nullptr; }
int32_t *i32(const Tensor &t) { return t.defined() ? static_cast<int32_t *>(t.data_ptr()) : nullptr; }
Tensor new_f32(at::IntArrayRef shape, const Call &c) { return at::empty(shape, at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, c.device)); }
Tensor new_i32(at::IntArrayRef shape, const Call &c) { return at::empty(shape, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, c.device)); }
void *stream_of(const Call &c) { return c10::cuda::getCurrentCUDAStream(c.device).stream(); }
void clear(const Call &c, const Tensor &a, const Tensor &b = Tensor(), const Tensor &d = Tensor()) {
    auto bytes = [](const Tensor &t) { return t.defined() ? 4 * t.numel() : 0; };
    check(lib.zero_buffers(f32(a), bytes(a), f32(b), bytes(b), f32(d), bytes(d), stream_of(c)));
}

// ------------------------------------------------------------------------------------------------ product mode's workspace
int64_t class_int(PyObject *name) {
    Ref v(PyObject_GetAttr(manager_base, name));
    int64_t n = 0;
    if (!v || !as_int(v.get(), n)) raise_current();
    return n;
}

// (data pointer, version, elements) of a tensor, as the manager's _histogram_key has them
PyObject *ident(const Tensor &t) {
    if (!t.defined()) Py_RETURN_NONE;
    return Py_BuildValue("(KkL)", (unsigned long long)(uintptr_t)t.data_ptr(), (unsigned long)t._version(), (long long)t.numel());
}
PyObject *histogram_key(const Call &c, int64_t B, const Tensor &x, const Tensor &pe, double eps, int variant) {
    Ref ix(ident(x)), ia(ident(c.anchors)), ip(ident(pe));
    return Py_BuildValue("(LLOOOOLLOdiK)", (long long)B, (long long)c.S, ix.get(), ix.get(), ia.get(), ip.get(), (long long)(x.numel() / (B * c.S)),
                         (long long)(x.numel() / (B * c.S)), c.cfg.sliced_product ? Py_True : Py_False, eps, variant,
                         (unsigned long long)(uintptr_t)stream_of(c));
}
// What the manager's _kept_histogram holds: (workspace, key, what was counted).  The memory the key names stays taken as long as the
// key can be found, so that no other call's inputs can lie there.
PyObject *kept_entry(const Call &c, const Tensor &workspace, PyObject *key, const Tensor &x, const Tensor &pe) {
    Ref t(THPVariable_Wrap(workspace)), tx(THPVariable_Wrap(x.detach())), ta(THPVariable_Wrap(c.anchors.detach())),
        tp(pe.defined() ? THPVariable_Wrap(pe.detach()) : Py_NewRef(Py_None));
    if (!t || !tx || !ta || !tp) return nullptr;
    return Py_BuildValue("(OO(OOOO))", t.get(), key, tx.get(), tx.get(), ta.get(), tp.get());
}
double context_eps(const Call &c) {
    return PyFloat_AsDouble(item(instance_dict(item(c.dict, names.shared_context)), names.cmp_eps));
}

// bytes of scratch of one call, as the manager's _product_scratch_bytes has them; 0: none
size_t product_scratch_bytes(const Call &c, int64_t B, bool backward, int variant) {
    const int64_t rows = (int64_t)1 << c.cfg.n_anchors;
    if (variant == LUTB_PRODUCT_DIRECT || c.S < 2 || (variant == LUTB_PRODUCT_AUTO && 4 * c.S < rows)) return 0;
    const size_t one = lib.product_workspace(&c.cfg, 1, (int32_t)c.S, backward), all = lib.product_workspace(&c.cfg, B, (int32_t)c.S, backward);
    return std::min(all, std::max(one, (size_t)std::max<int64_t>(0, class_int(names.scratch_limit))));
}
Tensor new_bytes(size_t bytes, const Call &c) {
    return bytes ? at::empty({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, c.device)) : Tensor();
}

int product_variant(const Call &c) {
    PyObject *v = item(c.dict, names.product_variant);
    int64_t n = 0;
    if (v == nullptr) return _PyType_Lookup(Py_TYPE(c.layer), names.product_variant) == nullptr ? 0 : -1;
    return as_int(v, n) ? (int)n : -1;
}

// ------------------------------------------------------------------------------------------------ backward
// Python's collector cannot look into a node in C++: one that owned its layer would keep a layer that holds on to its own output
// for ever.  So it knows the layer weakly, and owns what a layer that looks the same is made of (the parameters, the manager, the
// settings), for a backward pass that comes after the layer has gone.  (A node in Python, torch.autograd.Function's, costs 11 us a call.)
struct LayerNode : public torch::autograd::Node {
    PyObject *layer_ref, *cls;       // owned: weak reference, class
    std::vector<PyObject *> parts;   // owned, or null; by layer_parts
    Mode mode;
    std::vector<SavedVariable> saved;

    LayerNode(PyObject *layer, PyObject *ref, PyObject *dict, Mode m) : layer_ref(ref), cls(Py_NewRef((PyObject *)Py_TYPE(layer))), mode(m) {
        parts.reserve(layer_parts.size());
        for (PyObject *name : layer_parts) parts.push_back(Py_XNewRef(item(dict, name)));
    }
    ~LayerNode() override {
        if (Py_IsInitialized()) {
            pybind11::gil_scoped_acquire gil;
            Py_CLEAR(layer_ref);
            Py_CLEAR(cls);
            for (PyObject *&p : parts) Py_CLEAR(p);
        }
    }
    // The layer, or one made of its parts (a new reference; null with an exception)
    PyObject *layer() const {
        PyObject *alive = PyWeakref_GetObject(layer_ref);   // (borrowed; None: gone)
        if (alive == nullptr) return nullptr;
        if (alive != Py_None) return Py_NewRef(alive);
        Ref args(PyTuple_New(0)), dict(PyDict_New());
        if (!args || !dict) return nullptr;
        for (size_t i = 0; i < parts.size(); i++)
            if (parts[i] != nullptr && PyDict_SetItem(dict.get(), layer_parts[i], parts[i]) != 0) return nullptr;
        PyTypeObject *type = reinterpret_cast<PyTypeObject *>(cls);
        Ref made(type->tp_new(type, args.get(), nullptr));
        if (!made || PyObject_SetAttrString(made.get(), "__dict__", dict.get()) != 0) return nullptr;
        return Py_NewRef(made.get());
    }
    std::string name() const override { return "_LUTFunctionBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto &s : saved) s.reset_data();
    }
    std::vector<Tensor> unpack() {
        std::vector<Tensor> s;
        std::lock_guard<std::mutex> lock(mutex_);
        s.reserve(saved.size());
        for (auto &v : saved) s.push_back(v.unpack());
        return s;
    }
    variable_list apply(variable_list &&grads) override;
};

// y.grad_fn.saved_tensors
PyObject *saved_tensors(PyObject *self, void *) {
    HANDLE_TH_ERRORS
    auto *node = dynamic_cast<LayerNode *>(reinterpret_cast<torch::autograd::THPCppFunction *>(self)->cdata.get());
    TORCH_CHECK(node != nullptr, "not the node of a layer call");
    const std::vector<Tensor> s = node->unpack();
    Ref t(PyTuple_New((Py_ssize_t)s.size()));
    if (!t) return nullptr;
    for (size_t i = 0; i < s.size(); i++) PyTuple_SET_ITEM(t.get(), (Py_ssize_t)i, THPVariable_Wrap(s[i]));
    return Py_NewRef(t.get());
    END_HANDLE_TH_ERRORS
}
// y.grad_fn.layer
PyObject *node_layer(PyObject *self, void *) {
    HANDLE_TH_ERRORS
    auto *node = dynamic_cast<LayerNode *>(reinterpret_cast<torch::autograd::THPCppFunction *>(self)->cdata.get());
    TORCH_CHECK(node != nullptr, "not the node of a layer call");
    return node->layer();
    END_HANDLE_TH_ERRORS
}

// The layer's Python method, on the saved tensors: everything the native route does not take.
variable_list python_backward(LayerNode &node, PyObject *layer_obj, const std::vector<Tensor> &saved, const Tensor &dy, bool need_dx) try {
    namespace py = pybind11;
    py::object layer = py::reinterpret_borrow<py::object>(layer_obj), none = py::none();
    auto obj = [&](size_t i) { return i < saved.size() ? py::cast(saved[i]) : none; };
    py::object r;
    if (node.mode == NONSEQ)
        r = layer.attr("backward_step")(obj(0), py::cast(dy), obj(1), obj(2), obj(3), py::arg("need_input_grad") = need_dx);
    else if (node.mode == CONCAT)
        r = layer.attr("backward_step_concat")(obj(0), py::cast(dy), obj(1), obj(2), obj(3), obj(4), obj(5), obj(6));
    else
        r = layer.attr("backward_step_product")(obj(0), obj(1), py::cast(dy));
    variable_list out(node.num_outputs());
    py::tuple t = r;
    for (size_t i = 0; i < t.size() && i < out.size(); i++)
        if (!t[i].is_none()) out[i] = t[i].cast<Tensor>();
    return out;
} catch (pybind11::error_already_set &e) {
    e.restore();
    raise_current();   // (the engine hands Python's own exception on to the caller of backward)
}

// The Sparse policy's list straight from the table-gradient pass: fully connected non-sequence layers, unless switched off.
bool rows_direct(const Call &c) {
    return c.mode == NONSEQ && c.fully_connected && item(c.dict, names.sparse_rows_direct) == nullptr &&
           _PyType_Lookup(Py_TYPE(c.layer), names.sparse_rows_direct) == Py_True;
}

// What the manager's table_gradient_cells does, as a sparse tensor; undefined where no cell is touched.
Tensor sparse_table_gradient(const Call &c, int64_t B, const Tensor &dy, const Tensor &idx) {
    const int64_t O = c.cfg.n_outputs, capacity = std::min<int64_t>(B, (int64_t)1 << c.cfg.n_anchors) * c.cfg.n_detectors;
    const auto on = at::TensorOptions().device(at::kCUDA, c.device);
    auto bytes = [&](size_t n) { return at::empty({(int64_t)n}, on.dtype(at::kByte)); };
    const size_t rows_need = lib.rows_workspace(&c.cfg, B), cells_need = lib.cells_workspace(capacity * O);
    const Tensor ws = bytes(rows_need), ws2 = bytes(cells_need), ids = at::empty({capacity}, on.dtype(at::kLong)),
                 values = new_f32({capacity * O}, c), counts = at::empty({2}, on.dtype(at::kLong));
    int64_t *ids_p = static_cast<int64_t *>(ids.data_ptr()), *count = static_cast<int64_t *>(counts.data_ptr()), *total = count + 1;
    check(lib.rows(&c.cfg, B, f32(dy), i32(idx), ids_p, f32(values), capacity, count, ws.data_ptr(), rows_need, stream_of(c)));
    check(lib.cells_count(f32(values), count, capacity, (int32_t)O, total, ws2.data_ptr(), cells_need, stream_of(c)));
    int64_t n;
    {
        pybind11::gil_scoped_release others;
        n = counts.select(0, 1).item<int64_t>();
    }
    if (n == 0) return Tensor();
    const Tensor cells = at::empty({1, n}, on.dtype(at::kLong)), out = new_f32({n}, c);
    check(lib.cells_scatter(f32(values), ids_p, count, capacity, (int32_t)O, static_cast<int64_t *>(cells.data_ptr()), f32(out), n, ws2.data_ptr(),
                            cells_need, stream_of(c)));
    return at::_sparse_coo_tensor_unsafe(cells, out, c.weights.sizes(), at::TensorOptions().dtype(at::kFloat).layout(at::kSparse).device(at::kCUDA, c.device),
                                         true);
}

variable_list LayerNode::apply(variable_list &&grads) {
    std::vector<Tensor> s = unpack();
    const bool need_dx = task_should_compute_output(0);
    Tensor dy = grads[0];
    pybind11::gil_scoped_acquire gil;
    Ref layer_obj(layer());
    if (!layer_obj) raise_current();
    const Tensor &x = s[0];
    if (!dy.defined()) {   // an output nobody used: zeros, as torch hands them to a Python function
        const auto &m = input_metadata(0);
        dy = at::zeros_symint(m.shape_as_dim_vector(), m.options());
    }
    Call c;
    const bool readable = ordinary_context() && read_layer(layer_obj.get(), c, true);
    if (!readable) PyErr_Clear();
    bool native = readable && c.mode == mode && !c.normalized &&
                  (c.policy_type == policy_dense || c.policy_type == policy_internal || (c.policy_type == policy_sparse && rows_direct(c))) && is_true(item(c.dm_dict, names.dm_forward_seen));
    for (size_t i = 0; native && i < s.size(); i++) {
        const bool ints = mode != PRODUCT && (i == 1 || i == 3 || i == 4 || i == 6);
        native = plain_cuda(s[i], ints ? at::kInt : at::kFloat, c.device);
    }
    native = native && plain_cuda(dy, at::kFloat, c.device);
    int64_t dw_variant = 0;
    native = native && as_int(item(c.dict, names.dw_variant), dw_variant) && (mode != PRODUCT || product_variant(c) >= 0);
    if (!native) return python_backward(*this, layer_obj.get(), s, dy, need_dx);
    at::NoGradGuard no_grad;   // (results carry no graph either way: their values come from kernels)
    c10::cuda::CUDAGuard guard(c.device);
    const Tensor xc = x.contiguous(), dyc = dy.contiguous();
    const int64_t B = x.dim() > 0 ? x.size(0) : 0;
    const bool internal = c.policy_type == policy_internal, listed = c.policy_type == policy_sparse;
    // shapes: the saved tensors could come from a hook, the gradient from anywhere
    const int64_t Nt = c.cfg.n_detectors, tokens = B * c.S;
    bool fits = B > 0 && dy.numel() == tokens * c.cfg.n_outputs && x.dim() >= 2 && x.size(1) == c.S;
    if (mode != PRODUCT) {
        fits = fits && xc.numel() == tokens * c.cfg.n_inputs;
        for (size_t i = 1; i < s.size(); i++) {
            fits = fits && s[i].numel() == (i <= 3 ? tokens : c.S - 1) * Nt;
            s[i] = s[i].contiguous();
        }
        fits = fits && s.size() == (size_t)(mode == CONCAT && c.npe > 0 ? 7 : 4);
    } else {
        fits = fits && s.size() == (size_t)(c.npe > 0 ? 2 : 1) && (c.npe == 0 || s[1].numel() == (c.S - 1) * Nt * c.npe);
    }
    if (!fits) return python_backward(*this, layer_obj.get(), s, dy, need_dx);
    double lr = -1.0;
    if (internal) {
        Ref r(PyObject_CallMethodNoArgs(layer_obj.get(), names.external_lr));
        if (!r) raise_current();
        lr = PyFloat_AsDouble(r.get());
        if (lr == -1.0 && PyErr_Occurred()) raise_current();
    }
    Tensor dx, dw, dpe;
    if (listed) lr = LUTB_SKIP_TABLE_GRADIENT;   // (the list has its own pass)
    else if (!internal) dw = new_f32(c.weights.sizes(), c);
    float *target = f32(dw);
    if (mode == NONSEQ) {
        if (need_dx) dx = new_f32(x.sizes(), c);
        if (c.fully_connected) {
            if (need_dx) dw_variant |= LUTB_DX_WRITE;   // (written, not added to)
            if (dw.defined()) clear(c, dw);
            if (listed && !need_dx) return {dx, sparse_table_gradient(c, B, dyc, s[1])};
            const size_t need = lib.fc_backward_workspace(&c.cfg, B, (int)dw_variant);
            Tensor ws;
            if (need) ws = at::empty({(int64_t)need}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, c.device));
            check(lib.fc_backward(&c.cfg, B, f32(c.weights), f32(dyc), i32(c.anchors), i32(s[1]), f32(s[2]), i32(s[3]), f32(dx), target, lr,
                                  (int)dw_variant, need ? ws.data_ptr() : nullptr, need, stream_of(c)));
            if (listed) dw = sparse_table_gradient(c, B, dyc, s[1]);
        } else {
            clear(c, dx, dw);
            check(lib.sparse_backward(&c.cfg, &c.sparse, B, f32(c.weights), f32(dyc), i32(c.anchors), i32(s[1]), f32(s[2]), i32(s[3]), f32(dx),
                                      target, lr, stream_of(c)));
        }
        return {dx, dw};
    }
    dx = new_f32(x.sizes(), c);
    if (mode == CONCAT) {
        const bool pos = c.npe > 0;
        if (pos) dpe = new_f32({(c.S - 1) * Nt * c.npe}, c);
        clear(c, dx, dw, dpe);
        auto at_ = [&](size_t i) { return i < s.size() ? s[i] : Tensor(); };
        check(lib.concat_backward(&c.cfg, B, f32(c.weights), f32(dyc), i32(c.anchors), i32(s[1]), f32(s[2]), i32(s[3]), i32(at_(4)), f32(at_(5)),
                                  i32(at_(6)), f32(dx), f32(dpe), target, lr, stream_of(c)));
        return pos ? variable_list{dx, dw, dpe} : variable_list{dx, dw};
    }
    const Tensor pe = c.npe > 0 ? s[1].detach().contiguous().view(-1) : Tensor();
    if (pe.defined()) dpe = new_f32({pe.numel()}, c);
    clear(c, dx, dw, dpe);
    int variant = product_variant(c);
    const int64_t e = xc.numel() / tokens;
    Ref kept(Py_XNewRef(item(c.dm_dict, names.dm_kept)));
    PyDict_SetItem(c.dm_dict, names.dm_kept, Py_None);
    Tensor ws;
    int flags = 0;
    if (kept && PyTuple_Check(kept.get()) && PyTuple_GET_SIZE(kept.get()) == 3) {
        Ref key(histogram_key(c, B, xc, pe, context_eps(c), variant));
        const int same = key ? PyObject_RichCompareBool(PyTuple_GET_ITEM(kept.get(), 1), key.get(), Py_EQ) : -1;
        if (same < 0) raise_current();
        // the forward pass over these very inputs left its histogram in this workspace
        if (same == 1 && exact_tensor(PyTuple_GET_ITEM(kept.get(), 0))) {
            ws = THPVariable_Unpack(PyTuple_GET_ITEM(kept.get(), 0));
            flags = LUTB_PRODUCT_REUSE_HIST;
        }
    }
    if (!flags) ws = new_bytes(product_scratch_bytes(c, B, true, variant), c);
    check(lib.product_backward(&c.cfg, B, (int32_t)c.S, f32(c.weights), f32(xc), f32(xc), (int32_t)e, (int32_t)e, f32(pe), i32(c.anchors),
                               f32(dyc), f32(dx), f32(dx), f32(dpe), target, lr, variant | flags, ws.defined() ? ws.data_ptr() : nullptr,
                               ws.defined() ? (size_t)ws.numel() : 0, stream_of(c)));
    return pe.defined() ? variable_list{dx, dw, dpe} : variable_list{dx, dw};
}

// ------------------------------------------------------------------------------------------------ forward
PyObject *apply(PyObject *x_obj, PyObject *layer) {
    if (!exact_tensor(x_obj) || !ordinary_context()) Py_RETURN_NONE;
    const Tensor x = THPVariable_Unpack(x_obj);
    Call c;
    if (!read_layer(layer, c, false)) {
        if (PyErr_Occurred()) PyErr_Clear();
        Py_RETURN_NONE;
    }
    if (!plain_cuda(x, at::kFloat, c.device) || x.is_inference() || c.weights.is_inference()) Py_RETURN_NONE;
    const bool graph = at::GradMode::is_enabled();
    // (a layer in evaluation mode that is asked for gradients: the Python function has the answer)
    if (x._fw_grad(0).defined() || c.weights._fw_grad(0).defined()) Py_RETURN_NONE;

    std::vector<int64_t> in_shape, out_shape;
    if (x.dim() < 2 || !append_shape(layer, names.input_shape, in_shape) || (int64_t)in_shape.size() + 2 != x.dim()) Py_RETURN_NONE;
    for (size_t i = 0; i < in_shape.size(); i++)
        if (x.size((int64_t)i + 2) != in_shape[i]) Py_RETURN_NONE;
    const int64_t B = x.size(0), S = c.S, Nt = c.cfg.n_detectors;
    if (B <= 0 || x.size(1) != S) Py_RETURN_NONE;
    out_shape = {B, S};
    if (!append_shape(layer, names.output_shape, out_shape)) Py_RETURN_NONE;
    int64_t outputs = 1, inputs = 1;
    for (size_t i = 2; i < out_shape.size(); i++) outputs *= out_shape[i];
    for (int64_t n : in_shape) inputs *= n;
    if (outputs != c.cfg.n_outputs || inputs != (c.mode == PRODUCT ? (c.cfg.n_inputs - c.npe) / 2 : c.cfg.n_inputs)) Py_RETURN_NONE;
    const int variant = c.mode == PRODUCT ? product_variant(c) : 0;
    if (variant < 0) Py_RETURN_NONE;

    // positional embeddings of sequence layers, with their own graph where they are shared by the detectors
    Tensor pe_in, pe;
    if (c.mode != NONSEQ) {
        PyObject *p = item(item(c.dict, names.dict_parameters), names.positional);
        if (c.npe > 0) {
            if (!exact_tensor(p)) Py_RETURN_NONE;
            if (is_true(item(c.dict, names.unified))) {
                Ref r(PyObject_CallMethodNoArgs(layer, names.prepare_positional));
                if (!r) raise_current();
                if (!exact_tensor(r.get())) Py_RETURN_NONE;
                pe_in = THPVariable_Unpack(r.get());
            } else {
                pe_in = THPVariable_Unpack(p);
            }
            if (!plain_cuda(pe_in, at::kFloat, c.device) || pe_in.numel() != (S - 1) * Nt * c.npe || pe_in._fw_grad(0).defined() ||
                pe_in.is_inference())
                Py_RETURN_NONE;
        }
    }
    const bool needs_grad = graph && (x.requires_grad() || c.weights.requires_grad() || (pe_in.defined() && pe_in.requires_grad()));
    if (needs_grad && !c.training) Py_RETURN_NONE;

    Tensor out;
    std::vector<Tensor> saved;
    {
        at::NoGradGuard no_grad;
        c10::cuda::CUDAGuard guard(c.device);
        const Tensor xc = x.contiguous();
        out = new_f32(out_shape, c);
        clear(c, out);
        Tensor idx, md, mk, pidx, pmd, pmk;
        if (c.mode != PRODUCT) {
            idx = new_i32({B, S, Nt}, c);
            if (c.training) {
                md = new_f32({B, S, Nt}, c);
                mk = new_i32({B, S, Nt}, c);
            }
        }
        if (pe_in.defined()) pe = pe_in.detach().contiguous().view(-1);
        if (c.mode == NONSEQ) {
            if (c.fully_connected)
                check(lib.fc_forward(&c.cfg, B, f32(c.weights), f32(xc), i32(c.anchors), f32(out), i32(idx), f32(md), i32(mk), stream_of(c)));
            else
                check(lib.sparse_forward(&c.cfg, &c.sparse, B, f32(c.weights), f32(xc), i32(c.anchors), f32(out), i32(idx), f32(md), i32(mk),
                                         stream_of(c)));
        } else if (c.mode == CONCAT) {
            if (pe.defined()) {
                pidx = new_i32({S - 1, Nt}, c);
                if (c.training) {
                    pmd = new_f32({S - 1, Nt}, c);
                    pmk = new_i32({S - 1, Nt}, c);
                }
            }
            check(lib.concat_forward(&c.cfg, B, f32(c.weights), f32(xc), i32(c.anchors), f32(pe), f32(out), i32(idx), f32(md), i32(mk), i32(pidx),
                                     f32(pmd), i32(pmk), stream_of(c)));
        } else {
            PyDict_SetItem(c.dm_dict, names.dm_kept, Py_None);
            Tensor ws;
            const size_t scratch = product_scratch_bytes(c, B, false, variant);
            int flags = 0;
            if (c.training && scratch > 0) {
                // training: the row histogram is left in a workspace of its own for the backward pass
                const size_t want = lib.product_workspace(&c.cfg, B, (int32_t)S, 1);
                if (want > 0 && (int64_t)want <= class_int(names.keep_limit)) {
                    const Tensor own = new_bytes(want, c);
                    if (lib.product_keeps_histogram(&c.cfg, B, (int32_t)S, (int32_t)inputs, (int32_t)inputs, variant, own.data_ptr(), want)) {
                        Ref key(histogram_key(c, B, xc, pe, context_eps(c), variant));
                        Ref entry(key ? kept_entry(c, own, key.get(), xc, pe) : nullptr);
                        if (!entry) raise_current();
                        PyDict_SetItem(c.dm_dict, names.dm_kept, entry.get());
                        ws = own;
                        flags = LUTB_PRODUCT_KEEP_HIST;
                    }
                }
            }
            if (!flags) ws = new_bytes(scratch, c);
            check(lib.product_forward(&c.cfg, B, (int32_t)S, f32(c.weights), f32(xc), f32(xc), (int32_t)inputs, (int32_t)inputs, f32(pe),
                                      i32(c.anchors), f32(out), variant | flags, ws.defined() ? ws.data_ptr() : nullptr,
                                      ws.defined() ? (size_t)ws.numel() : 0, stream_of(c)));
        }
        PyDict_SetItem(c.dm_dict, names.dm_forward_seen, Py_True);
        if (needs_grad) {
            saved = {x};
            if (c.mode != PRODUCT) saved.insert(saved.end(), {idx, md, mk});
            if (c.mode == CONCAT && pidx.defined()) saved.insert(saved.end(), {pidx, pmd, pmk});
            if (c.mode == PRODUCT && pe_in.defined()) saved.push_back(pe_in);
        }
    }
    if (needs_grad) {
        PyObject *ref = PyWeakref_NewRef(layer, nullptr);
        if (ref == nullptr) raise_current();
        auto node = std::shared_ptr<LayerNode>(new LayerNode(layer, ref, c.dict, c.mode), torch::autograd::deleteNode);
        node->set_next_edges(pe_in.defined() ? torch::autograd::collect_next_edges(x, c.weights, pe_in)
                                             : torch::autograd::collect_next_edges(x, c.weights));
        for (const Tensor &t : saved) node->saved.emplace_back(t, false);
        torch::autograd::set_history(out, node);
    }
    return THPVariable_Wrap(out);
}

PyObject *apply_entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n == 2, "apply(x, layer)");
    return apply(args[0], args[1]);
    END_HANDLE_TH_ERRORS
}

void setup(pybind11::dict addresses, pybind11::object layer_cls, pybind11::object manager_cls, pybind11::object base_cls, pybind11::object dense,
           pybind11::object internal, pybind11::object sparse, pybind11::object check_fn, pybind11::list layer_names, pybind11::list hook_names, pybind11::list manager_names,
           pybind11::list part_names) {
    auto take = [&](const char *name, auto &fn) { fn = reinterpret_cast<std::decay_t<decltype(fn)>>(addresses[name].cast<uintptr_t>()); };
    take("lutb_nonseq_fc_forward", lib.fc_forward);
    take("lutb_nonseq_fc_backward", lib.fc_backward);
    take("lutb_nonseq_fc_backward_workspace", lib.fc_backward_workspace);
    take("lutb_nonseq_sparse_forward", lib.sparse_forward);
    take("lutb_nonseq_sparse_backward", lib.sparse_backward);
    take("lutb_concat_forward", lib.concat_forward);
    take("lutb_concat_backward", lib.concat_backward);
    take("lutb_product_forward", lib.product_forward);
    take("lutb_product_backward", lib.product_backward);
    take("lutb_product_workspace", lib.product_workspace);
    take("lutb_product_keeps_histogram", lib.product_keeps_histogram);
    take("lutb_zero_buffers", lib.zero_buffers);
    take("lutb_nonseq_fc_table_grad_rows", lib.rows);
    take("lutb_nonseq_fc_table_grad_rows_workspace", lib.rows_workspace);
    take("lutb_dense_to_sparse_workspace", lib.cells_workspace);
    take("lutb_row_cells_count", lib.cells_count);
    take("lutb_row_cells_scatter", lib.cells_scatter);
    auto keep = [](pybind11::object o) { return o.release().ptr(); };   // for the life of the process
    layer_class = keep(layer_cls);
    manager_class = keep(manager_cls);
    manager_base = keep(base_cls);
    policy_dense = keep(dense);
    policy_internal = keep(internal);
    policy_sparse = keep(sparse);
    check_status = keep(check_fn);
    tensor_class = keep(pybind11::module_::import("torch").attr("Tensor"));
    parameter_class = keep(pybind11::module_::import("torch.nn").attr("Parameter"));
    auto in = [](const char *s) { return PyUnicode_InternFromString(s); };
    names = Names{in("_parameters"), in("_buffers"), in("_weights"), in("_detector_anchors"), in("_positional_embeddings"), in("training"), in("_lut_dm"),
                  in("_shared_context"), in("_cmp_eps"), in("device"), in("_weights_gradient_policy"), in("type"), in("normalized"), in("_sequence_length"),
                  in("_concatenation_product"), in("_sliced_product_mode"), in("_positional_dim"), in("_unified_positional_embeddings"),
                  in("_is_fully_connected"), in("_dw_variant"), in("_product_variant"), in("_sparse_rows_direct"), in("_device"),
                  in("_fully_connected"), in("_sparse"), in("_seq_len"), in("_forward_seen"), in("_kept_histogram"), in("n_weights"),
                  in("_rows_per_detector"), in("_cfg"), in("c_struct"), in("input_shape"), in("output_shape"), in("_prepare_positional_embeddings"),
                  in("_external_lr"), in("product_scratch_limit"), in("product_keep_limit")};
    auto originals = [&](PyObject *cls, pybind11::list list, std::vector<std::pair<PyObject *, PyObject *>> &out) {
        for (auto n : list) {
            PyObject *name = in(n.cast<std::string>().c_str());
            PyObject *fn = _PyType_Lookup(reinterpret_cast<PyTypeObject *>(cls), name);
            TORCH_CHECK(fn != nullptr, "no method ", n.cast<std::string>());
            out.emplace_back(name, Py_NewRef(fn));
        }
    };
    originals(layer_class, layer_names, layer_methods);
    originals(manager_class, manager_names, manager_methods);
    for (auto n : hook_names) layer_hooks.push_back(in(n.cast<std::string>().c_str()));
    for (auto n : part_names) layer_parts.push_back(in(n.cast<std::string>().c_str()));
    using namespace torch::autograd;   // (as the macro wants it)
    static PyGetSetDef properties[] = {THP_FUNCTION_DEFAULT_PROPERTIES,
                                       {"saved_tensors", saved_tensors, nullptr, nullptr, nullptr},
                                       {"layer", node_layer, nullptr, nullptr, nullptr},
                                       {nullptr}};
    static PyTypeObject node_type;
    _initFunctionPyTypeObject(node_type, "_LUTFunctionBackward", properties, nullptr);
    registerCppFunction(typeid(LayerNode), &node_type);
}

PyMethodDef methods[] = {{"apply", (PyCFunction)(void (*)(void))apply_entry, METH_FASTCALL, "output of layer(x), or None"}, {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(_layer_calls, m) {
    m.def("setup", &setup);
    m.attr("torch_version") = TORCH_VERSION;
    PyModule_AddFunctions(m.ptr(), methods);
}
