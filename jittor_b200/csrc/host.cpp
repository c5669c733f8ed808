// Native host path: the Var / Op objects of the lazy graph and the replay of planned graphs.
//
// What bounded it before: a graph was matched, fused and launched by Python on every sync -- 0.1 ms for a softmax and its
// gradient, 3 ms for a convolution + BatchNorm + ReLU block with its gradients, whose kernels take 0.35 ms. A program runs the
// same few graphs over and over with other tensors, so the first sync of a graph runs the Python planner with every
// allocation and library call written to a tape (executor.py), and later syncs of a graph of the same structure replay that
// tape from here: one walk over the graph makes its signature (op kinds, attributes, shapes, dtypes, how nodes share
// inputs, alignment of the leaves and which of them share memory), a hash lookup finds the tape, and its calls run with the
// new pointers. Results are not kept: every replay allocates its outputs and launches every kernel again.
#include <Python.h>
#include <structmember.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <deque>
#include <memory>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "../../include/b200jt.h"

namespace {

// ------------------------------------------------------------------------------------------------ hooks set by the package
PyObject *h_shape_type, *h_make_shape, *h_dtype_type, *h_canon, *h_record, *h_error, *h_flags;
PyObject *s_running_mean, *s_running_var, *s_momentum, *s_wait, *s_sig, *s_also, *s_custom, *s_fuse, *s_wgrad, *s_collective, *s_value;
long g_context = 0;          // host state that changes plans (SMs reserved for a collective): part of every signature
bool g_recording = false;
int64_t g_plans = 0, g_replays = 0, g_records = 0;
const char* (*g_last_error)() = nullptr;

inline bool none(PyObject* o) { return o == nullptr || o == Py_None; }

// ------------------------------------------------------------------------------------------------ Op
struct OpObj {
    PyObject_HEAD
    PyObject *kind, *inputs, *attrs;
};

int op_init(OpObj* self, PyObject* args, PyObject* kw) {
    PyObject *kind, *inputs;
    if (!PyArg_ParseTuple(args, "OO", &kind, &inputs)) return -1;
    PyObject* list = PySequence_List(inputs);
    if (!list) return -1;
    PyObject* attrs = kw ? PyDict_Copy(kw) : PyDict_New();
    if (!attrs) { Py_DECREF(list); return -1; }
    Py_INCREF(kind);
    Py_XSETREF(self->kind, kind);
    Py_XSETREF(self->inputs, list);
    Py_XSETREF(self->attrs, attrs);
    return 0;
}
int op_traverse(OpObj* self, visitproc visit, void* arg) {
    Py_VISIT(self->inputs);
    Py_VISIT(self->attrs);
    return 0;
}
int op_clear(OpObj* self) {
    Py_CLEAR(self->kind);
    Py_CLEAR(self->inputs);
    Py_CLEAR(self->attrs);
    return 0;
}
void op_dealloc(OpObj* self) {
    PyObject_GC_UnTrack(self);
    Py_TRASHCAN_BEGIN(self, op_dealloc)
    op_clear(self);
    Py_TYPE(self)->tp_free((PyObject*)self);
    Py_TRASHCAN_END
}
PyMemberDef op_members[] = {
    {"kind", T_OBJECT, offsetof(OpObj, kind), 0, nullptr},
    {"inputs", T_OBJECT, offsetof(OpObj, inputs), 0, nullptr},
    {"attrs", T_OBJECT, offsetof(OpObj, attrs), 0, nullptr},
    {nullptr}};
PyTypeObject OpType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ------------------------------------------------------------------------------------------------ Var
struct VarObj {
    PyObject_HEAD
    PyObject *shape, *dtype, *op, *builder, *data, *name, *konst, *pending, *options, *relay, *vjp, *bn_running;
    char is_scalar, stop_grad, stop_fuse;
};
PyTypeObject VarType = {PyVarObject_HEAD_INIT(nullptr, 0)};
inline bool is_var(PyObject* o) { return PyObject_TypeCheck(o, &VarType); }

// What Var's make_shape and canon make of their argument. Lists and tuples of plain whole numbers are copied here, and the names of
// dtypes are asked for once: a layer's call makes a dozen of each.
PyObject* shape_from(PyObject* x) {
    const bool list = PyList_CheckExact(x);
    if (!list && !PyTuple_CheckExact(x)) return PyObject_CallOneArg(h_make_shape, x);
    const Py_ssize_t n = list ? PyList_GET_SIZE(x) : PyTuple_GET_SIZE(x);
    auto item = [&](Py_ssize_t i) { return list ? PyList_GET_ITEM(x, i) : PyTuple_GET_ITEM(x, i); };
    bool plain = n <= B200JT_MAX_DIMS;
    for (Py_ssize_t i = 0; plain && i < n; i++) plain = PyLong_CheckExact(item(i));
    if (!plain) return PyObject_CallOneArg(h_make_shape, x);
    PyTypeObject* t = (PyTypeObject*)h_shape_type;
    PyObject* s = t->tp_alloc(t, 0);
    for (Py_ssize_t i = 0; s && i < n; i++) if (PyList_Append(s, item(i)) < 0) Py_CLEAR(s);
    return s;
}
PyObject* dtype_from(PyObject* x) {
    static PyObject* known = PyDict_New();
    if (!PyUnicode_CheckExact(x)) return PyObject_CallOneArg(h_canon, x);
    if (PyObject* d = PyDict_GetItemWithError(known, x)) return Py_NewRef(d);
    if (PyErr_Occurred()) return nullptr;
    PyObject* d = PyObject_CallOneArg(h_canon, x);
    if (d && PyDict_SetItem(known, x, d) < 0) Py_CLEAR(d);
    return d;
}

int var_init(VarObj* self, PyObject* args, PyObject* kw) {
    static const char* names[] = {"shape", "dtype", "op", "data", "is_scalar", nullptr};
    PyObject *shape, *dtype, *op = Py_None, *data = Py_None;
    int scalar = 0;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "OO|OOp", (char**)names, &shape, &dtype, &op, &data, &scalar)) return -1;
    if ((PyObject*)Py_TYPE(shape) == h_shape_type) Py_INCREF(shape);
    else if (!(shape = shape_from(shape))) return -1;
    if ((PyObject*)Py_TYPE(dtype) == h_dtype_type) Py_INCREF(dtype);
    else if (!(dtype = dtype_from(dtype))) { Py_DECREF(shape); return -1; }
    Py_XSETREF(self->shape, shape);
    Py_XSETREF(self->dtype, dtype);
    Py_INCREF(op);
    Py_XSETREF(self->op, op);
    Py_INCREF(data);
    Py_XSETREF(self->data, data);
    self->is_scalar = (char)scalar;
    return 0;
}
int var_traverse(VarObj* self, visitproc visit, void* arg) {
    Py_VISIT(self->shape); Py_VISIT(self->op); Py_VISIT(self->builder); Py_VISIT(self->data); Py_VISIT(self->konst);
    Py_VISIT(self->pending); Py_VISIT(self->options); Py_VISIT(self->relay); Py_VISIT(self->vjp); Py_VISIT(self->bn_running);
    return 0;
}
int var_clear(VarObj* self) {
    Py_CLEAR(self->shape); Py_CLEAR(self->dtype); Py_CLEAR(self->op); Py_CLEAR(self->builder); Py_CLEAR(self->data);
    Py_CLEAR(self->name); Py_CLEAR(self->konst); Py_CLEAR(self->pending); Py_CLEAR(self->options); Py_CLEAR(self->relay);
    Py_CLEAR(self->vjp); Py_CLEAR(self->bn_running);
    return 0;
}
void var_dealloc(VarObj* self) {
    PyObject_GC_UnTrack(self);
    Py_TRASHCAN_BEGIN(self, var_dealloc)
    var_clear(self);
    Py_TYPE(self)->tp_free((PyObject*)self);
    Py_TRASHCAN_END
}
// A producer that is written down only when something reads it: `_builder` returns the Op on first access.
PyObject* var_get_op(VarObj* self, void*) {
    if (!none(self->builder)) {
        PyObject* b = self->builder;
        self->builder = nullptr;
        PyObject* op = PyObject_CallNoArgs(b);
        if (!op) {                                          // asked again it fails the same way
            if (none(self->builder)) Py_XSETREF(self->builder, b); else Py_DECREF(b);
            return nullptr;
        }
        Py_DECREF(b);
        Py_XSETREF(self->op, op);
    }
    return Py_NewRef(self->op ? self->op : Py_None);
}
int var_set_op(VarObj* self, PyObject* v, void*) {
    Py_CLEAR(self->builder);
    Py_XSETREF(self->op, Py_NewRef(v ? v : Py_None));
    return 0;
}
PyObject* var_get_options(VarObj* self, void*) {
    if (!self->options && !(self->options = PyDict_New())) return nullptr;
    return Py_NewRef(self->options);
}
int var_set_options(VarObj* self, PyObject* v, void*) {
    Py_XSETREF(self->options, Py_XNewRef(v));
    return 0;
}
PyMemberDef var_members[] = {
    {"_shape", T_OBJECT, offsetof(VarObj, shape), 0, nullptr}, {"_dtype", T_OBJECT, offsetof(VarObj, dtype), 0, nullptr},
    {"_data", T_OBJECT, offsetof(VarObj, data), 0, nullptr}, {"_name", T_OBJECT, offsetof(VarObj, name), 0, nullptr},
    {"_const", T_OBJECT, offsetof(VarObj, konst), 0, nullptr}, {"_pending", T_OBJECT, offsetof(VarObj, pending), 0, nullptr},
    {"_relay", T_OBJECT, offsetof(VarObj, relay), 0, nullptr}, {"_vjp", T_OBJECT, offsetof(VarObj, vjp), 0, nullptr},
    {"_bn_running", T_OBJECT, offsetof(VarObj, bn_running), 0, nullptr},
    {"_builder", T_OBJECT, offsetof(VarObj, builder), 0, nullptr},
    {"is_scalar", T_BOOL, offsetof(VarObj, is_scalar), 0, nullptr}, {"_stop_grad", T_BOOL, offsetof(VarObj, stop_grad), 0, nullptr},
    {"_stop_fuse", T_BOOL, offsetof(VarObj, stop_fuse), 0, nullptr},
    {"shape", T_OBJECT, offsetof(VarObj, shape), READONLY, nullptr}, {"size", T_OBJECT, offsetof(VarObj, shape), READONLY, nullptr},
    {"dtype", T_OBJECT, offsetof(VarObj, dtype), READONLY, nullptr},
    {nullptr}};
PyGetSetDef var_getset[] = {
    {"_op", (getter)var_get_op, (setter)var_set_op, nullptr, nullptr},
    {"compile_options", (getter)var_get_options, (setter)var_set_options, nullptr, nullptr},
    {nullptr}};

// ------------------------------------------------------------------------------------------------ signature of a graph
// Post-order walk over everything unrealised under the roots. Two graphs with the same key are planned the same way: the
// key holds whatever the planner can look at. `ok` is false for graphs the planner may not be skipped for (collectives,
// Python callables without a signature, leaves that are not plain CUDA tensors).
struct Walk {
    std::string key;
    std::vector<VarObj*> nodes, leaves;
    std::vector<PyObject*> held;                     // every Var met: Python that runs meanwhile (a builder, a wait, another thread) may drop it
    std::unordered_map<const void*, int> index;      // Var -> number: leaves and nodes share one numbering in visiting order
    std::vector<std::pair<size_t, size_t>> numbers;  // where the key holds the value of a Python number: (place, bytes)
    bool ok = true;
    int count = 0;

    Walk() = default;
    Walk(const Walk&) = delete;
    ~Walk() { for (PyObject* o : held) Py_DECREF(o); }
    void raw(const void* p, size_t n) { key.append((const char*)p, n); }
    void num(int64_t v) { raw(&v, sizeof v); }
    void tag(char c) { key.push_back(c); }
    void text(PyObject* s) {
        Py_ssize_t n;
        const char* c = PyUnicode_AsUTF8AndSize(s, &n);
        if (!c) { PyErr_Clear(); ok = false; return; }
        tag('s'); num(n); raw(c, (size_t)n);
    }
    void value(PyObject* v) {
        if (v == Py_None) tag('n');
        else if (v == Py_True) tag('t');
        else if (v == Py_False) tag('f');
        else if (PyLong_Check(v)) { tag('i'); num(PyLong_AsLongLong(v)); if (PyErr_Occurred()) { PyErr_Clear(); ok = false; } }
        else if (PyFloat_Check(v)) { double d = PyFloat_AS_DOUBLE(v); tag('d'); raw(&d, sizeof d); }
        else if (PyUnicode_Check(v)) text(v);
        else if (PyTuple_Check(v)) { tag('('); num(PyTuple_GET_SIZE(v)); for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(v); i++) value(PyTuple_GET_ITEM(v, i)); }
        else if (PyList_Check(v)) { tag('('); num(PyList_GET_SIZE(v)); for (Py_ssize_t i = 0; i < PyList_GET_SIZE(v); i++) value(PyList_GET_ITEM(v, i)); }
        else if (is_var(v)) { tag('v'); num(index.count(v) ? index[v] : -1); }
        else ok = false;
    }
    void number(PyObject* v) {
        const size_t at = key.size();
        value(v);
        if (key.size() > at + 1) numbers.emplace_back(at + 1, key.size() - at - 1);       // what kind of number it is stays
    }
    // the key with every number the same
    std::string skeleton() const {
        std::string k = key;
        for (auto& n : numbers) std::fill_n(k.begin() + n.first, n.second, '\0');
        return k;
    }
    void meta(VarObj* v) {
        PyObject* s = v->shape;
        if (!s || !PyList_Check(s)) { ok = false; return; }
        const Py_ssize_t n = PyList_GET_SIZE(s);
        tag((char)('A' + n));
        for (Py_ssize_t i = 0; i < n; i++) num(PyLong_AsLongLong(PyList_GET_ITEM(s, i)));
        text(v->dtype);
        if (!none(v->konst)) { tag('c'); number(v->konst); }
        tag((char)(v->stop_fuse * 2 + v->is_scalar));
    }
    static void vars_in(PyObject* t, std::vector<VarObj*>& out) {
        if (is_var(t)) out.push_back((VarObj*)t);
        else if (PyTuple_Check(t)) for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(t); i++) vars_in(PyTuple_GET_ITEM(t, i), out);
        else if (PyList_Check(t)) for (Py_ssize_t i = 0; i < PyList_GET_SIZE(t); i++) vars_in(PyList_GET_ITEM(t, i), out);
    }
    void leaf(VarObj* v) {
        tag('L');
        meta(v);
        if (!THPVariable_Check(v->data)) { ok = false; return; }
        const at::Tensor& t = THPVariable_Unpack(v->data);
        if (!t.is_cuda() || !t.is_contiguous()) { ok = false; return; }
        const uintptr_t p = (uintptr_t)t.const_data_ptr();
        tag((char)(p % 16 == 0 ? 2 : p % 8 == 0 ? 1 : 0));
        tag((char)t.device().index());
        tag((char)t.scalar_type());
        num(t.numel());
        leaves.push_back(v);
    }
    // children of an unrealised Var, in the order the key refers to them
    void children(VarObj* v, std::vector<VarObj*>& out) {
        if (!none(v->relay)) vars_in(v->relay, out);
        else {
            PyObject* op = var_get_op(v, nullptr);
            if (!op) { PyErr_Clear(); ok = false; return; }
            Py_DECREF(op);                                    // v->op keeps it
            if (none(op) || Py_TYPE(op) != &OpType) { ok = false; return; }
            OpObj* o = (OpObj*)op;
            vars_in(o->inputs, out);
            if (PyObject* also = PyDict_GetItem(o->attrs, s_also)) vars_in(also, out);
        }
        if (!none(v->bn_running)) {
            PyObject* t = v->bn_running;                      // (module, batch mean, batch variance)
            if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 3) { ok = false; return; }
            for (PyObject* name : {s_running_mean, s_running_var}) {
                PyObject* r = PyObject_GetAttr(PyTuple_GET_ITEM(t, 0), name);
                if (!r || !is_var(r)) { PyErr_Clear(); Py_XDECREF(r); ok = false; return; }
                out.push_back((VarObj*)r);
                Py_DECREF(r);                                 // the module keeps it
            }
            vars_in(t, out);
        }
    }
    void node(VarObj* v) {
        tag('N');
        meta(v);
        if (!none(v->relay)) value(v->relay);
        else {
            OpObj* o = (OpObj*)v->op;
            text(o->kind);
            if (PyUnicode_Compare(o->kind, s_collective) == 0) { ok = false; return; }
            PyObject* sig = PyDict_GetItem(o->attrs, s_sig);
            if (sig) value(sig);
            else if (PyUnicode_Compare(o->kind, s_custom) == 0) { ok = false; return; }
            else {
                Py_ssize_t pos = 0;
                PyObject *k, *x;
                while (PyDict_Next(o->attrs, &pos, &k, &x)) { text(k); if (k == s_value) number(x); else value(x); }
            }
            value(o->inputs);
            if (PyObject* also = PyDict_GetItem(o->attrs, s_also)) value(also);
        }
        if (!none(v->bn_running)) {
            PyObject* t = v->bn_running;
            PyObject* m = PyTuple_GET_ITEM(t, 0);
            tag('B');
            PyObject* mom = PyObject_GetAttr(m, s_momentum);
            if (!mom) { PyErr_Clear(); ok = false; return; }
            value(mom);
            Py_DECREF(mom);
            for (PyObject* name : {s_running_mean, s_running_var}) {
                PyObject* r = PyObject_GetAttr(m, name);
                value(r);
                Py_DECREF(r);
            }
            value(PyTuple_GET_ITEM(t, 1));
            value(PyTuple_GET_ITEM(t, 2));
        }
        nodes.push_back(v);
    }
    void flag(PyObject* name) {
        PyObject* f = PyDict_GetItem(h_flags, name);
        if (f) value(f);
    }
    // A tape knows a leaf by its addresses: leaves that share memory (assign, a realised reshape, two Vars of one torch tensor)
    // and leaves that do not are different graphs. For each leaf that starts inside another one: which, and how far in. That
    // fixes every address of a group of overlapping leaves relative to the others'.
    void sharing() {
        struct Span { uintptr_t at, end; size_t leaf; };
        std::vector<Span> spans;
        spans.reserve(leaves.size());
        for (size_t i = 0; i < leaves.size(); i++) {
            const at::Tensor& t = THPVariable_Unpack(leaves[i]->data);
            const uintptr_t at = (uintptr_t)t.const_data_ptr();
            if (t.numel()) spans.push_back({at, at + (size_t)t.numel() * t.element_size(), i});
        }
        std::sort(spans.begin(), spans.end(), [](const Span& a, const Span& b) { return a.at != b.at ? a.at < b.at : a.leaf < b.leaf; });
        Span last{0, 0, 0};                      // the span that reaches furthest so far
        for (const Span& s : spans) {
            if (s.at < last.end) { tag('o'); num((int64_t)s.leaf); num((int64_t)last.leaf); num((int64_t)(s.at - last.at)); }
            if (s.end > last.end) last = s;
        }
    }
    void run(const std::vector<VarObj*>& roots) {
        key.reserve(1 << 13);                            // a training step of a small network is 150 nodes and 10 KB
        index.reserve(256);
        held.reserve(256);
        nodes.reserve(128);
        flag(s_fuse); flag(s_wgrad);
        num(g_context);
        if (c10::cuda::device_count() < 1) { ok = false; return; }
        tag((char)c10::cuda::current_device());
        struct Frame { VarObj* v; std::vector<VarObj*> kids; size_t next; };
        std::vector<Frame> stack;
        for (VarObj* root : roots) {
            if (!index.count(root)) { index.emplace(root, -1); stack.push_back({root, {}, 0}); }
            while (ok && !stack.empty()) {
                Frame& f = stack.back();
                if (f.next == 0 && f.kids.empty() && none(f.v->data)) {
                    children(f.v, f.kids);
                    for (VarObj* k : f.kids) held.push_back(Py_NewRef((PyObject*)k));
                }
                if (!ok) break;
                if (f.next < f.kids.size()) {
                    VarObj* k = f.kids[f.next++];
                    if (index.emplace(k, -1).second) stack.push_back({k, {}, 0});
                    continue;
                }
                if (none(f.v->data)) node(f.v); else leaf(f.v);
                index[f.v] = count++;
                stack.pop_back();
            }
            tag('r'); num(index[root]);
        }
        if (ok) sharing();
    }
};

// ------------------------------------------------------------------------------------------------ tapes
union Slot { void* p; int64_t i; double d; };
template <class A> inline A slot_as(const Slot& s) {
    if constexpr (std::is_pointer_v<A>) return reinterpret_cast<A>(s.p);
    else if constexpr (std::is_floating_point_v<A>) return (A)s.d;
    else return (A)s.i;
}
template <class F> struct Inv;
template <class R, class... A> struct Inv<R (*)(A...)> {
    template <size_t... I> static int64_t go(void* fn, const Slot* s, std::index_sequence<I...>) {
        return (int64_t)reinterpret_cast<R (*)(A...)>(fn)(slot_as<A>(s[I])...);
    }
    static int64_t call(void* fn, const Slot* s) { return go(fn, s, std::index_sequence_for<A...>{}); }
};
typedef int64_t (*Invoke)(void*, const Slot*);
struct Entry { const char* name; Invoke invoke; void* fn; };
#define E(name) {#name, &Inv<decltype(&name)>::call, nullptr}
Entry g_entries[] = {
    E(b200jt_reindex), E(b200jt_reindex_reduce_workspace), E(b200jt_reindex_reduce), E(b200jt_setitem), E(b200jt_broadcast_to),
    E(b200jt_reduce_workspace), E(b200jt_reduce), E(b200jt_binary), E(b200jt_unary), E(b200jt_ternary), E(b200jt_fused_chain),
    E(b200jt_softmax), E(b200jt_softmax_backward), E(b200jt_layer_norm), E(b200jt_matmul_workspace), E(b200jt_matmul_least_workspace), E(b200jt_matmul),
    E(b200jt_batched_matmul), E(b200jt_conv2d_workspace), E(b200jt_conv2d), E(b200jt_conv2d_formats_workspace), E(b200jt_conv2d_formats),
    E(b200jt_conv2d_transpose), E(b200jt_conv2d_backward_w), E(b200jt_conv2d_backward_w_workspace), E(b200jt_conv2d_backward_w_tc),
    E(b200jt_conv2d_backward_w_formats_workspace), E(b200jt_conv2d_backward_w_formats), E(b200jt_bn_stats), E(b200jt_bn_apply),
    E(b200jt_layer_norm_backward_workspace), E(b200jt_layer_norm_backward), E(b200jt_bn_backward_sums),
    E(b200jt_bn_backward_dx), E(b200jt_bn_backward), E(b200jt_pool2d), E(b200jt_pool2d_backward), E(b200jt_pool2d_backward_indices), E(b200jt_pool2d_taps), E(b200jt_conv2d_backward_x), E(b200jt_conv2d_backward_x_workspace),
    E(b200jt_pool2d_backward_taps),
};
#undef E
Entry* entry_of(const char* name) {
    for (Entry& e : g_entries) if (std::strcmp(e.name, name) == 0 && e.fn) return &e;
    return nullptr;
}

struct Patch { void** where; int buf; int64_t off; };
struct Step {
    enum Kind { ALLOC, WORKSPACE, CALL, FILL } kind;
    int buf = -1;                          // ALLOC, WORKSPACE, FILL: the buffer
    std::vector<int64_t> sizes;            // ALLOC
    at::ScalarType type = at::kByte;       // ALLOC
    double value = 0;                      // FILL
    Entry* entry = nullptr;                // CALL, WORKSPACE
    Entry* least = nullptr;                // WORKSPACE: what the call cannot do without, where it takes less than it asks for
    std::vector<Slot> slots;
    std::vector<Patch> patches;
    std::vector<std::pair<int, int>> nbytes;   // (slot, buffer): the size of a workspace passed beside its pointer
    int stream = -1;                       // slot of the stream
    std::string what;                      // CALL: what an error is reported as
    std::vector<int> release;              // buffers nothing reads after this step
    std::vector<int> moved;                // CALL: nodes whose running statistics it moves; a later step may fail, and they move once
};
struct Result { int node, buf; bool same; int64_t off; std::vector<int64_t> shape; size_t ready; };      // ready: steps after which it has its value
struct Tape {
    int n_leaves = 0, n_bufs = 0, n_plans = 0;
    std::vector<Step> steps;
    std::vector<Result> results;
    // storage behind the slots
    std::deque<std::vector<b200jt_tensor>> tensors;
    std::deque<std::string> strings;
    std::deque<std::vector<const char*>> string_lists;
    std::deque<std::vector<int64_t>> longs;
    std::deque<std::vector<int32_t>> ints;
};
// null: the planner has to run every time. Shared: a replay keeps its tape while another thread clears the map.
typedef std::unordered_map<std::string, std::shared_ptr<Tape>> Tapes;
// Programs with endless shapes fill the map: when the newer half is full it becomes the older one, whose tapes are dropped
// unless they were used since. A number that changes from call to call (a learning rate) makes a graph of its own each time,
// which is not worth a record: after kMaxVariants of a structure that differ in their numbers only, others are planned.
constexpr size_t kHalf = 2048;
constexpr int kMaxVariants = 16;
Tapes g_tapes, g_older;
std::unordered_map<std::string, int> g_variants;
void age_tapes() {
    if (g_variants.size() >= 2 * kHalf) g_variants.clear();
    if (g_tapes.size() < kHalf) return;
    g_older = std::move(g_tapes);
    g_tapes.clear();
    g_variants.clear();
}
const std::shared_ptr<Tape>* find_tape(const std::string& key) {
    auto it = g_tapes.find(key);
    if (it != g_tapes.end()) return &it->second;
    auto old = g_older.find(key);
    if (old == g_older.end()) return nullptr;
    std::shared_ptr<Tape> tape = std::move(old->second);
    g_older.erase(old);
    age_tapes();
    return &g_tapes.emplace(key, std::move(tape)).first->second;
}

// One argument of a recorded call: (code, payload...), written by _capi.Recorder.
bool add_arg(Tape& t, Step& st, PyObject* a) {
    const char* code = PyUnicode_AsUTF8(PyTuple_GET_ITEM(a, 0));
    if (!code) return false;
    Slot s; s.p = nullptr;
    const int at = (int)st.slots.size();
    st.slots.push_back(s);
    auto arg = [&](Py_ssize_t k) { return PyTuple_GET_ITEM(a, k); };
    switch (code[0]) {
        case '0': break;
        case 'z': st.stream = at; break;
        case 'i': st.slots[at].i = PyLong_AsLongLong(arg(1)); break;
        case 'd': st.slots[at].d = PyFloat_AsDouble(arg(1)); break;
        case 'n': st.nbytes.emplace_back(at, (int)PyLong_AsLong(arg(1))); break;
        case 'p': st.patches.push_back({nullptr, (int)PyLong_AsLong(arg(1)), PyLong_AsLongLong(arg(2))});
                  st.patches.back().where = (void**)(intptr_t)(-1 - at); break;          // resolved once the slots stop moving
        case 'b': {
            char* c; Py_ssize_t n;
            if (PyBytes_AsStringAndSize(arg(1), &c, &n) < 0) return false;
            t.strings.emplace_back(c, (size_t)n);
            st.slots[at].p = (void*)t.strings.back().c_str();
            break;
        }
        case 'T': {                                                                   // [(dtype, shape, buffer, offset), ...]
            PyObject* list = arg(1);
            const Py_ssize_t n = PyList_GET_SIZE(list);
            t.tensors.emplace_back((size_t)(n > 0 ? n : 1));
            auto& v = t.tensors.back();
            std::memset(v.data(), 0, v.size() * sizeof(b200jt_tensor));
            for (Py_ssize_t i = 0; i < n; i++) {
                PyObject* d = PyList_GET_ITEM(list, i);
                PyObject* shape = PyTuple_GET_ITEM(d, 1);
                v[i].dtype = (int32_t)PyLong_AsLong(PyTuple_GET_ITEM(d, 0));
                v[i].ndim = (int32_t)PyTuple_GET_SIZE(shape);
                for (int j = 0; j < v[i].ndim; j++) v[i].shape[j] = PyLong_AsLongLong(PyTuple_GET_ITEM(shape, j));
                const int buf = (int)PyLong_AsLong(PyTuple_GET_ITEM(d, 2));
                if (buf >= 0) st.patches.push_back({&v[i].ptr, buf, PyLong_AsLongLong(PyTuple_GET_ITEM(d, 3))});
            }
            st.slots[at].p = v.data();
            break;
        }
        case 'S': {
            PyObject* list = arg(1);
            const Py_ssize_t n = PyList_GET_SIZE(list);
            t.string_lists.emplace_back();
            auto& v = t.string_lists.back();
            for (Py_ssize_t i = 0; i < n; i++) {
                t.strings.emplace_back(PyBytes_AsString(PyList_GET_ITEM(list, i)));
                v.push_back(t.strings.back().c_str());
            }
            v.push_back(nullptr);
            st.slots[at].p = (void*)v.data();
            break;
        }
        case 'q': case 'w': {
            PyObject* list = arg(1);
            const Py_ssize_t n = PyList_GET_SIZE(list);
            if (code[0] == 'q') {
                t.longs.emplace_back();
                for (Py_ssize_t i = 0; i < n; i++) t.longs.back().push_back(PyLong_AsLongLong(PyList_GET_ITEM(list, i)));
                st.slots[at].p = t.longs.back().data();
            } else {
                t.ints.emplace_back();
                for (Py_ssize_t i = 0; i < n; i++) t.ints.back().push_back((int32_t)PyLong_AsLong(PyList_GET_ITEM(list, i)));
                st.slots[at].p = t.ints.back().data();
            }
            break;
        }
        default: PyErr_Format(PyExc_RuntimeError, "tape: unknown argument code %s", code); return false;
    }
    return !PyErr_Occurred();
}

bool ints_of(PyObject* tuple, std::vector<int64_t>& out) {
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(tuple); i++) out.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(tuple, i)));
    return !PyErr_Occurred();
}

// spec: (number of buffers, steps, results, (step, node) whose running statistics move, plans) from executor._record
std::shared_ptr<Tape> build_tape(PyObject* spec, int n_leaves) {
    PyObject *steps, *results, *bn;
    auto t = std::make_shared<Tape>();
    if (!PyArg_ParseTuple(spec, "iO!O!O!i", &t->n_bufs, &PyList_Type, &steps, &PyList_Type, &results, &PyList_Type, &bn, &t->n_plans))
        return nullptr;
    t->n_leaves = n_leaves;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(steps); i++) {
        PyObject* s = PyList_GET_ITEM(steps, i);
        const char* kind = PyUnicode_AsUTF8(PyTuple_GET_ITEM(s, 0));
        if (!kind) return nullptr;
        t->steps.emplace_back();
        Step& st = t->steps.back();
        if (!std::strcmp(kind, "alloc")) {
            st.kind = Step::ALLOC;
            st.buf = (int)PyLong_AsLong(PyTuple_GET_ITEM(s, 1));
            if (!ints_of(PyTuple_GET_ITEM(s, 2), st.sizes)) return nullptr;
            st.type = (at::ScalarType)PyLong_AsLong(PyTuple_GET_ITEM(s, 3));
        } else if (!std::strcmp(kind, "fill")) {
            st.kind = Step::FILL;
            st.buf = (int)PyLong_AsLong(PyTuple_GET_ITEM(s, 1));
            st.value = PyFloat_AsDouble(PyTuple_GET_ITEM(s, 2));
        } else {
            st.kind = kind[0] == 'w' ? Step::WORKSPACE : Step::CALL;
            st.buf = (int)PyLong_AsLong(PyTuple_GET_ITEM(s, 1));
            const char* name = PyUnicode_AsUTF8(PyTuple_GET_ITEM(s, 2));
            if (!name || !(st.entry = entry_of(name))) return nullptr;
            if (!std::strcmp(name, "b200jt_matmul_workspace")) st.least = entry_of("b200jt_matmul_least_workspace");
            PyObject* args = PyTuple_GET_ITEM(s, 3);
            st.slots.reserve((size_t)PyList_GET_SIZE(args));
            for (Py_ssize_t k = 0; k < PyList_GET_SIZE(args); k++) if (!add_arg(*t, st, PyList_GET_ITEM(args, k))) return nullptr;
            if (st.kind == Step::CALL) {
                const char* what = PyUnicode_AsUTF8(PyTuple_GET_ITEM(s, 4));
                if (!what) return nullptr;
                st.what = what;
            }
        }
        if (PyErr_Occurred()) return nullptr;
    }
    for (Step& st : t->steps)
        for (Patch& p : st.patches)
            if ((intptr_t)p.where < 0) p.where = &st.slots[(size_t)(-1 - (intptr_t)p.where)].p;
    std::vector<char> kept((size_t)t->n_bufs, 0);
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(results); i++) {
        PyObject* r = PyList_GET_ITEM(results, i);
        Result out;
        out.node = (int)PyLong_AsLong(PyTuple_GET_ITEM(r, 0));
        out.buf = (int)PyLong_AsLong(PyTuple_GET_ITEM(r, 1));
        out.off = PyLong_AsLongLong(PyTuple_GET_ITEM(r, 2));
        if (!ints_of(PyTuple_GET_ITEM(r, 3), out.shape)) return nullptr;
        out.ready = PyLong_AsSize_t(PyTuple_GET_ITEM(r, 4));
        out.same = false;
        // the buffer is allocated in its result's shape, so that no view is needed for it
        if (out.off == 0 && out.buf >= n_leaves && !kept[out.buf])
            for (Step& st : t->steps)
                if (st.kind == Step::ALLOC && st.buf == out.buf) {
                    int64_t a = 1, b = 1;
                    for (int64_t d : st.sizes) a *= d;
                    for (int64_t d : out.shape) b *= d;
                    if (a == b) { st.sizes = out.shape; out.same = true; }
                }
        kept[out.buf] = 1;
        t->results.push_back(std::move(out));
    }
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(bn); i++) {
        PyObject* m = PyList_GET_ITEM(bn, i);
        const size_t step = PyLong_AsSize_t(PyTuple_GET_ITEM(m, 0));
        if (step >= t->steps.size()) return nullptr;
        t->steps[step].moved.push_back((int)PyLong_AsLong(PyTuple_GET_ITEM(m, 1)));
    }
    std::vector<int> last((size_t)t->n_bufs, -1);
    for (size_t k = 0; k < t->steps.size(); k++) {
        Step& st = t->steps[k];
        if (st.buf >= 0) last[st.buf] = (int)k;
        for (Patch& p : st.patches) last[p.buf] = (int)k;
        for (auto& n : st.nbytes) last[n.second] = (int)k;
    }
    for (int b = n_leaves; b < t->n_bufs; b++)
        if (!kept[b] && last[b] >= 0) t->steps[last[b]].release.push_back(b);
    if (PyErr_Occurred()) return nullptr;
    return t;
}

// Buffers belong to the call. Slots and descriptors belong to the tape: a step writes its own and is launched with the
// interpreter lock held all the while, so that two threads in one tape do not see each other's.
bool replay(Tape& t, const Walk& w) {
    std::vector<at::Tensor> bufs((size_t)t.n_bufs);
    for (int i = 0; i < t.n_leaves; i++) bufs[i] = THPVariable_Unpack(w.leaves[i]->data);
    // Hands out what the first `steps` steps have computed. Where a step fails, what was computed before it stays, as in the
    // planner: running statistics among it, which moved and are not moved again.
    auto hand_out = [&](size_t steps) {
        for (const Result& r : t.results) {
            if (r.ready > steps) continue;
            at::Tensor out = bufs[r.buf];
            if (!r.same) {
                int64_t n = 1;
                for (int64_t d : r.shape) n *= d;
                if (r.off == 0 && n == out.numel()) out = out.view(r.shape);
                else {
                    std::vector<int64_t> stride(r.shape.size(), 1);
                    for (int i = (int)r.shape.size() - 2; i >= 0; i--) stride[i] = stride[i + 1] * r.shape[i + 1];
                    out = out.as_strided(r.shape, stride, out.storage_offset() + r.off / (int64_t)out.element_size());
                }
            }
            PyObject* py = THPVariable_Wrap(std::move(out));
            if (!py) return false;
            Py_XSETREF(w.nodes[r.node]->data, py);
        }
        return true;
    };
    const auto device = c10::Device(c10::kCUDA, c10::cuda::current_device());
    void* stream = (void*)c10::cuda::getCurrentCUDAStream().stream();
    size_t at = 0;
    try {
        for (; at < t.steps.size(); at++) {
            Step& st = t.steps[at];
            if (st.kind == Step::ALLOC) {
                bufs[st.buf] = at::Tensor(at::detail::empty_cuda(st.sizes, st.type, device, std::nullopt));
                continue;
            }
            if (st.kind == Step::FILL) { bufs[st.buf].fill_(st.value); continue; }
            for (Patch& p : st.patches) {
                const at::Tensor& b = bufs[p.buf];
                *p.where = b.defined() ? (char*)b.data_ptr() + p.off : nullptr;
            }
            for (auto& n : st.nbytes) st.slots[n.first].i = bufs[n.second].defined() ? bufs[n.second].numel() : 0;
            if (st.stream >= 0) st.slots[st.stream].p = stream;
            int64_t rc = st.entry->invoke(st.entry->fn, st.slots.data());
            if (st.kind == Step::WORKSPACE) {
                auto get = [&] { if (rc > 0) bufs[st.buf] = at::Tensor(at::detail::empty_cuda({rc}, at::kByte, device, std::nullopt)); };
                if (!st.least) get();
                else {
                    bool room = true;
                    try { get(); } catch (const c10::OutOfMemoryError&) { room = false; }
                    if (!room) { rc = st.least->invoke(st.least->fn, st.slots.data()); get(); }
                }
            } else if (rc != 0) {
                const std::string why = g_last_error ? g_last_error() : "";
                if (hand_out(at)) PyErr_Format(h_error, "%s: %s (status %d)", st.what.c_str(), why.c_str(), (int)rc);
                return false;
            }
            for (int n : st.moved) Py_XSETREF(w.nodes[n]->bn_running, Py_NewRef(Py_None));
            for (int b : st.release) bufs[b].reset();
        }
    } catch (...) {
        if (!hand_out(at)) return false;
        throw;
    }
    if (!hand_out(t.steps.size())) return false;
    g_plans += t.n_plans;
    g_replays++;
    return true;
}

// ------------------------------------------------------------------------------------------------ building the graph
// What an expression costs before anything runs: shape and dtype inference and a node per op. The rules are the Python
// ones (var.py, dtypes.py), which are asked once per (op, dtypes, flags) and remembered.
PyObject *h_var_type, *h_infer_binary, *h_infer_unary, *h_infer_reduce, *h_to_var, *h_op_grad;
PyObject* h_dtypes[10];                         // DType objects by code
PyObject *k_binary, *k_unary, *k_ternary, *k_reduce, *k_fill, *k_broadcast, *k_reshape, *k_reindex, *k_op, *k_value, *k_mask, *k_keep, *k_rmask,
    *s_amp, *o_add, *o_subtract, *o_multiply, *o_divide, *o_maximum, *o_minimum, *o_equal, *o_negative, *o_mean, *o_log, *o_exp, *i_zero;
enum { BOOL, INT8, INT16, INT32, INT64, UINT8, F16, BF16, F32, F64 };

int dtype_code(PyObject* s) {
    for (int i = 0; i < 10; i++) if (h_dtypes[i] == s) return i;
    for (int i = 0; i < 10; i++) if (PyUnicode_Compare(h_dtypes[i], s) == 0) return i;
    return -1;
}
inline bool is_float(int d) { return d >= F16; }
inline bool is_half(int d) { return d == F16 || d == BF16; }
inline long amp() {
    PyObject* a = PyDict_GetItem(h_flags, s_amp);
    return a ? PyLong_AsLong(a) : 0;
}
struct Ref {                                     // owned reference
    PyObject* p;
    Ref(PyObject* o = nullptr) : p(o) {}
    Ref(Ref&& r) : p(r.p) { r.p = nullptr; }
    Ref& operator=(Ref&& r) { PyObject* o = r.p; r.p = nullptr; Py_XSETREF(p, o); return *this; }
    Ref(const Ref&) = delete;
    ~Ref() { Py_XDECREF(p); }
    PyObject* give() { PyObject* o = p; p = nullptr; return o; }
    explicit operator bool() const { return p != nullptr; }
};
inline VarObj* V(PyObject* o) { return (VarObj*)o; }
inline Py_ssize_t rank_of(PyObject* v) { return PyList_GET_SIZE(V(v)->shape); }
inline int64_t dim_of(PyObject* v, Py_ssize_t i) { return PyLong_AsLongLong(PyList_GET_ITEM(V(v)->shape, i)); }
int64_t numel_of(PyObject* v) {
    int64_t n = 1;
    for (Py_ssize_t i = 0; i < rank_of(v); i++) n *= dim_of(v, i);
    return n;
}
bool same_shape(PyObject* a, PyObject* b) {
    if (V(a)->shape == V(b)->shape) return true;
    if (rank_of(a) != rank_of(b)) return false;
    for (Py_ssize_t i = 0; i < rank_of(a); i++) if (dim_of(a, i) != dim_of(b, i)) return false;
    return true;
}
PyObject* make_shape(const int64_t* d, size_t n) {
    PyTypeObject* t = (PyTypeObject*)h_shape_type;
    PyObject* s = t->tp_alloc(t, 0);
    if (!s) return nullptr;
    for (size_t i = 0; i < n; i++) {
        Ref v(PyLong_FromLongLong(d[i]));
        if (!v || PyList_Append(s, v.p) < 0) { Py_DECREF(s); return nullptr; }
    }
    return s;
}
// shape and op are taken over
PyObject* new_var(PyObject* shape, int dtype, PyObject* op, bool scalar = false) {
    PyTypeObject* t = (PyTypeObject*)h_var_type;
    VarObj* v = shape && op ? (VarObj*)t->tp_alloc(t, 0) : nullptr;
    if (!v) { Py_XDECREF(shape); Py_XDECREF(op); return nullptr; }
    v->shape = shape;
    v->dtype = Py_NewRef(h_dtypes[dtype]);
    v->op = op;
    v->data = Py_NewRef(Py_None);
    v->is_scalar = scalar;
    return (PyObject*)v;
}
PyObject* new_op(PyObject* kind, std::initializer_list<PyObject*> inputs, std::initializer_list<std::pair<PyObject*, PyObject*>> attrs) {
    OpObj* o = (OpObj*)OpType.tp_alloc(&OpType, 0);
    if (!o) return nullptr;
    o->kind = Py_NewRef(kind);
    o->inputs = PyList_New((Py_ssize_t)inputs.size());
    o->attrs = PyDict_New();
    if (!o->inputs || !o->attrs) { Py_DECREF(o); return nullptr; }
    Py_ssize_t i = 0;
    for (PyObject* v : inputs) PyList_SET_ITEM(o->inputs, i++, Py_NewRef(v));
    for (auto& a : attrs) if (!a.second || PyDict_SetItem(o->attrs, a.first, a.second) < 0) { Py_DECREF(o); return nullptr; }
    return (PyObject*)o;
}
PyObject* number_var(PyObject* value, int dtype) {               // a scalar made from a Python number
    const int64_t one = 1;
    PyObject* v = new_var(make_shape(&one, 1), dtype, new_op(k_fill, {}, {{k_value, value}}), true);
    if (v) V(v)->konst = Py_NewRef(value);
    return v;
}
PyObject* to_var(PyObject* x) {
    if (is_var(x)) return Py_NewRef(x);
    if (PyFloat_CheckExact(x)) return number_var(x, F32);
    if (PyBool_Check(x)) return number_var(x, BOOL);
    if (PyLong_CheckExact(x)) return number_var(x, INT32);
    return PyObject_CallOneArg(h_to_var, x);
}
PyObject* fill_like(PyObject* v, PyObject* value, int dtype) { return new_var(Py_NewRef(V(v)->shape), dtype, new_op(k_fill, {}, {{k_value, value}})); }

struct InferKey {
    const void* op;
    uint32_t rest;
    bool operator==(const InferKey& k) const { return op == k.op && rest == k.rest; }
};
struct InferHash { size_t operator()(const InferKey& k) const { return (size_t)(uintptr_t)k.op * 0x9e3779b97f4a7c15ull ^ (size_t)k.rest * 0x85ebca6bull; } };
std::unordered_map<InferKey, int, InferHash> g_infer;
int infer(PyObject* fn, PyObject* op, int x, int y, bool xs, bool ys) {
    if (x < 0 || y < 0) { PyErr_SetString(PyExc_ValueError, "unsupported dtype"); return -1; }
    PyObject* name = Py_NewRef(op);
    if (PyUnicode_CheckExact(name)) PyUnicode_InternInPlace(&name);
    Ref hold(name);
    const InferKey key{name, (uint32_t)((amp() & 63) << 16 | x << 12 | y << 8 | xs << 7 | ys << 6 | (fn == h_infer_binary ? 1 : fn == h_infer_unary ? 2 : 3))};
    auto it = g_infer.find(key);
    if (it != g_infer.end()) return it->second;
    Ref r(fn == h_infer_binary ? PyObject_CallFunction(fn, "OOOOO", op, h_dtypes[x], h_dtypes[y], xs ? Py_True : Py_False, ys ? Py_True : Py_False)
                               : PyObject_CallFunction(fn, "OO", op, h_dtypes[x]));
    if (!r) return -1;
    const int d = dtype_code(r.p);
    if (PyUnicode_CheckExact(name)) { Py_INCREF(name); g_infer.emplace(key, d); }       // the address stays this name's
    return d;
}

// the stretched shape of two operands (right-aligned, size-1 axes stretch); new reference, shared where it equals one of theirs
PyObject* stretched(PyObject* xs, PyObject* ys) {
    const Py_ssize_t nx = PyList_GET_SIZE(xs), ny = PyList_GET_SIZE(ys), n = nx > ny ? nx : ny;
    int64_t z[32];
    bool is_x = nx == n, is_y = ny == n;
    if (n > 32) { PyErr_SetString(PyExc_ValueError, "too many dims"); return nullptr; }
    for (Py_ssize_t i = 0; i < n; i++) {
        const int64_t a = i < n - nx ? 1 : PyLong_AsLongLong(PyList_GET_ITEM(xs, i - (n - nx))), b = i < n - ny ? 1 : PyLong_AsLongLong(PyList_GET_ITEM(ys, i - (n - ny)));
        if (a == b || b == 1) z[i] = a;
        else if (a == 1) z[i] = b;
        else { PyErr_Format(PyExc_ValueError, "Shape not match, x:%R y:%R", xs, ys); return nullptr; }
        is_x = is_x && z[i] == a;
        is_y = is_y && z[i] == b;
    }
    return is_x ? Py_NewRef(xs) : is_y ? Py_NewRef(ys) : make_shape(z, (size_t)n);
}

PyObject* binary(PyObject* a, PyObject* b, PyObject* op) {
    Ref x(to_var(a)), y(x ? to_var(b) : nullptr);
    if (!x || !y) return nullptr;
    const int d = infer(h_infer_binary, op, dtype_code(V(x.p)->dtype), dtype_code(V(y.p)->dtype), V(x.p)->is_scalar, V(y.p)->is_scalar);
    if (d < 0) return nullptr;
    PyObject* s = stretched(V(x.p)->shape, V(y.p)->shape);
    return s ? new_var(s, d, new_op(k_binary, {x.p, y.p}, {{k_op, op}})) : nullptr;
}
PyObject* unary(PyObject* a, PyObject* op) {
    Ref x(to_var(a));
    if (!x) return nullptr;
    const int dx = dtype_code(V(x.p)->dtype), to = dtype_code(op);
    if (to >= 0 && to == dx) return x.give();
    const int d = to >= 0 ? to : infer(h_infer_unary, op, dx, 0, false, false);
    if (d < 0) return nullptr;
    return new_var(Py_NewRef(V(x.p)->shape), d, new_op(k_unary, {x.p}, {{k_op, to >= 0 ? h_dtypes[to] : op}}), V(x.p)->is_scalar);
}
PyObject* ternary(PyObject* c0, PyObject* a, PyObject* b) {
    Ref c(to_var(c0)), x(c ? to_var(a) : nullptr), y(x ? to_var(b) : nullptr);
    if (!c || !x || !y) return nullptr;
    Ref z(stretched(V(c.p)->shape, V(x.p)->shape));
    if (!z) return nullptr;
    PyObject* s = stretched(z.p, V(y.p)->shape);
    if (!s) return nullptr;
    const int d = infer(h_infer_binary, o_add, dtype_code(V(x.p)->dtype), dtype_code(V(y.p)->dtype), V(x.p)->is_scalar, V(y.p)->is_scalar);
    if (d < 0) { Py_DECREF(s); return nullptr; }
    return new_var(s, d, new_op(k_ternary, {c.p, x.p, y.p}, {}));
}
PyObject* cast_to(PyObject* x, int d) { return unary(x, h_dtypes[d]); }
PyObject* reduce_masks(PyObject* x, PyObject* op, long mask, long keep) {
    int64_t z[32];
    size_t n = 0;
    for (Py_ssize_t i = 0; i < rank_of(x); i++) {
        if (!(mask >> i & 1)) z[n++] = dim_of(x, i);
        else if (keep >> i & 1) z[n++] = 1;
    }
    if (!n) z[n++] = 1;
    const int d = infer(h_infer_reduce, op, dtype_code(V(x)->dtype), 0, false, false);
    if (d < 0) return nullptr;
    Ref m(PyLong_FromLong(mask)), k(PyLong_FromLong(keep));
    return new_var(make_shape(z, n), d, new_op(k_reduce, {x}, {{k_op, op}, {k_rmask, m.p}, {k_keep, k.p}}));
}
PyObject* reshape_like(PyObject* g, PyObject* x) {
    if (same_shape(g, x)) return Py_NewRef(g);
    return new_var(Py_NewRef(V(x)->shape), dtype_code(V(g)->dtype), new_op(k_reshape, {g}, {}));
}
PyObject* bcast_like(PyObject* x, PyObject* ref, long mask, long keep) {
    Ref m(PyLong_FromLong(mask)), k(PyLong_FromLong(keep));
    return new_var(Py_NewRef(V(ref)->shape), dtype_code(V(x)->dtype), new_op(k_broadcast, {x}, {{k_mask, m.p}, {k_keep, k.p}}));
}
// jt.reduce: half inputs are summed in float32 unless amp_reg bit 32 is set
PyObject* reduce(PyObject* x0, PyObject* op, long mask, long keep) {
    Ref x(Py_NewRef(x0));
    const int d = dtype_code(V(x0)->dtype);
    const bool up = is_half(d) && !(amp() & 32) && (PyUnicode_Compare(op, o_add) == 0 || PyUnicode_Compare(op, o_mean) == 0);
    if (up) x = Ref(cast_to(x0, F32));
    if (!x) return nullptr;
    Ref r(reduce_masks(x.p, op, mask, keep));
    if (!r || !up) return r.give();
    return cast_to(r.p, d);
}

// ------------------------------------------------------------------------------------------------ reverse mode
// The per-op rules on the node constructors above; kinds that are rare stay in Python (grad.py, h_op_grad).
bool op_is(PyObject* name, PyObject* what) { return name == what || PyUnicode_Compare(name, what) == 0; }

// v is the constant 1 stretched to its shape (the seed of a gradient pushed through sums and casts)
bool is_ones(PyObject* v) {
    for (int i = 0; i < 8; i++) {
        VarObj* o = V(v);
        if (!none(o->data) || !none(o->builder) || none(o->op) || Py_TYPE(o->op) != &OpType) return false;
        OpObj* op = (OpObj*)o->op;
        if (op_is(op->kind, k_fill)) {
            PyObject* x = PyDict_GetItem(op->attrs, k_value);
            return x && !PyBool_Check(x) && ((PyLong_Check(x) && PyLong_AsLong(x) == 1) || (PyFloat_Check(x) && PyFloat_AS_DOUBLE(x) == 1.0));
        }
        if (!op_is(op->kind, k_broadcast)) {
            PyObject* name = op_is(op->kind, k_unary) ? PyDict_GetItem(op->attrs, k_op) : nullptr;
            if (!name || !is_float(dtype_code(name))) return false;
        }
        v = PyList_GET_ITEM(op->inputs, 0);
    }
    return false;
}

// sums g over the axes along which an operand of x's shape was stretched by a binary op
PyObject* unbroadcast(PyObject* g, PyObject* x) {
    if (same_shape(g, x)) return Py_NewRef(g);
    const Py_ssize_t pad = rank_of(g) - rank_of(x);
    long mask = 0;
    for (Py_ssize_t i = 0; i < rank_of(g); i++)
        if (i < pad || (dim_of(x, i - pad) == 1 && dim_of(g, i) != 1)) mask |= 1l << i;
    if (!mask) return reshape_like(g, x);
    Ref r(reduce(g, o_add, mask, (1l << rank_of(g)) - 1));
    return r ? reshape_like(r.p, x) : nullptr;
}

// gradient with respect to input k of the op that produced out; None where none flows
PyObject* op_grad(PyObject* out, PyObject* dout, Py_ssize_t k) {
    OpObj* o = (OpObj*)V(out)->op;
    PyObject* x = PyList_GET_ITEM(o->inputs, k);
    auto attr = [&](PyObject* name) { return PyDict_GetItem(o->attrs, name); };
    auto mask_of = [&](PyObject* name) { PyObject* m = attr(name); return m ? PyLong_AsLong(m) : 0l; };
    auto zeros = [&](PyObject* v) { return fill_like(v, i_zero, dtype_code(V(v)->dtype)); };
    if (op_is(o->kind, k_binary)) {
        PyObject *p = PyList_GET_ITEM(o->inputs, 0), *q = PyList_GET_ITEM(o->inputs, 1), *name = attr(k_op);
        Ref g;
        if (op_is(name, o_add)) g = Ref(Py_NewRef(dout));
        else if (op_is(name, o_subtract)) g = Ref(k == 0 ? Py_NewRef(dout) : unary(dout, o_negative));
        else if (op_is(name, o_multiply)) {
            // 1 * y is y bit for bit: the gradient of (p * q).sum() is the other factor itself, not a pass over it (not when the
            // factor is the reindex / broadcast operand of a convolution: its gradient graphs are recognised with the product)
            PyObject* other = k == 0 ? q : p;
            bool same = same_shape(other, dout) && op_is(V(other)->dtype, V(dout)->dtype) && is_float(dtype_code(V(other)->dtype)) && is_ones(dout);
            if (same && none(V(other)->builder) && !none(V(other)->op)) {
                PyObject* kind = ((OpObj*)V(other)->op)->kind;
                same = !op_is(kind, k_broadcast) && !op_is(kind, k_reindex);
            }
            g = Ref(same ? Py_NewRef(other) : binary(other, dout, o_multiply));
        } else if (op_is(name, o_divide)) {
            if (k == 0) g = Ref(binary(dout, q, o_divide));
            else {
                Ref n(unary(dout, o_negative)), np(n ? binary(n.p, p, o_multiply) : nullptr), qq(np ? binary(q, q, o_multiply) : nullptr);
                g = Ref(qq ? binary(np.p, qq.p, o_divide) : nullptr);
            }
        } else if (op_is(name, o_maximum) || op_is(name, o_minimum)) {
            Ref cond(binary(q, out, o_equal)), z(cond ? zeros(dout) : nullptr);
            g = Ref(z ? (k == 1 ? ternary(cond.p, dout, z.p) : ternary(cond.p, z.p, dout)) : nullptr);
        } else return PyObject_CallFunction(h_op_grad, "OOn", out, dout, k);
        return g ? unbroadcast(g.p, x) : nullptr;
    }
    if (op_is(o->kind, k_unary)) {
        PyObject* name = attr(k_op);
        const int dx = dtype_code(V(x)->dtype);
        if (!is_float(dx)) Py_RETURN_NONE;
        if (dtype_code(name) >= 0) return cast_to(dout, dx);
        if (op_is(name, o_negative)) return unary(dout, o_negative);
        if (op_is(name, o_log)) return binary(dout, x, o_divide);
        if (op_is(name, o_exp)) return binary(dout, out, o_multiply);
        return PyObject_CallFunction(h_op_grad, "OOn", out, dout, k);
    }
    if (op_is(o->kind, k_ternary)) {
        if (k == 0) Py_RETURN_NONE;
        PyObject* cond = PyList_GET_ITEM(o->inputs, 0);
        Ref z(zeros(dout)), g(z ? (k == 1 ? ternary(cond, dout, z.p) : ternary(cond, z.p, dout)) : nullptr);
        return g ? unbroadcast(g.p, x) : nullptr;
    }
    if (op_is(o->kind, k_reshape)) return reshape_like(dout, x);
    if (op_is(o->kind, k_broadcast)) {
        const long mask = mask_of(k_mask), keep = mask_of(k_keep);
        if (!mask) return Py_NewRef(dout);
        Ref g(reduce_masks(dout, o_add, mask, keep));
        return g ? reshape_like(g.p, x) : nullptr;
    }
    if (op_is(o->kind, k_reduce)) {
        const long mask = mask_of(k_rmask), keep = mask_of(k_keep);
        PyObject* name = attr(k_op);
        if (op_is(name, o_add)) return bcast_like(dout, x, mask, keep);
        if (op_is(name, o_mean)) {
            Ref b(bcast_like(dout, x, mask, keep)), f(PyFloat_FromDouble((double)numel_of(out) / (double)numel_of(x)));
            return b && f ? binary(b.p, f.p, o_multiply) : nullptr;
        }
    }
    return PyObject_CallFunction(h_op_grad, "OOn", out, dout, k);
}

// backprop(loss, dout, targets, through_graph) -> list of gradients, None where none arrives
PyObject* m_backprop(PyObject*, PyObject* args) {
    PyObject *loss, *dout0, *targets, *through;
    if (!PyArg_ParseTuple(args, "O!OO!O", &VarType, &loss, &dout0, &PyList_Type, &targets, &through)) return nullptr;
    struct Node { PyObject *v, *inputs; bool rule, need, target; };                    // inputs: a list or tuple the Var holds
    std::vector<Node> order;
    std::unordered_map<PyObject*, int> index;                                          // Var -> place in `order` (-1: on the stack)
    std::unordered_map<PyObject*, bool> wanted;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(targets); i++) {
        if (!is_var(PyList_GET_ITEM(targets, i))) { PyErr_SetString(PyExc_TypeError, "grad: targets must be Vars"); return nullptr; }
        wanted[PyList_GET_ITEM(targets, i)] = true;
    }
    struct Frame { PyObject *v, *inputs; bool rule; Py_ssize_t next; };
    std::vector<Frame> stack;
    // A rule that passes over a Var the program holds (its third element): the graph is followed where the gradient of that
    // Var is asked for, ends there, or another value was assigned to it.
    auto stops_inside = [&](PyObject* vjp) {
        if (PyTuple_GET_SIZE(vjp) < 3) return false;
        PyObject* inner = PyTuple_GET_ITEM(vjp, 2);
        return wanted.count(inner) > 0 || V(inner)->stop_grad || none(V(inner)->relay);
    };
    auto push = [&](PyObject* v) -> bool {
        Frame f{v, nullptr, false, 0};
        if (!wanted.count(v) && !V(v)->stop_grad) {                                    // no gradient flows through stop_grad Vars
            if (!none(V(v)->vjp) && v != through && !stops_inside(V(v)->vjp)) { f.inputs = PyTuple_GET_ITEM(V(v)->vjp, 0); f.rule = true; }
            else {
                PyObject* op = var_get_op(V(v), nullptr);
                if (!op) return false;
                Py_DECREF(op);                                                         // v keeps it
                if (!none(op)) f.inputs = ((OpObj*)op)->inputs;
            }
        }
        index[v] = -1;
        stack.push_back(f);
        return true;
    };
    auto count = [](PyObject* in) { return !in ? 0 : PyTuple_Check(in) ? PyTuple_GET_SIZE(in) : PyList_GET_SIZE(in); };
    auto item = [](PyObject* in, Py_ssize_t i) { return PyTuple_Check(in) ? PyTuple_GET_ITEM(in, i) : PyList_GET_ITEM(in, i); };
    if (!push(loss)) return nullptr;
    while (!stack.empty()) {
        const size_t top = stack.size() - 1;
        const Py_ssize_t n = count(stack[top].inputs);
        if (stack[top].next < n) {
            PyObject* i = item(stack[top].inputs, n - 1 - stack[top].next++);
            if (!index.count(i) && !push(i)) return nullptr;
            continue;
        }
        const Frame f = stack[top];
        const bool target = wanted.count(f.v) > 0;
        bool need = target;
        for (Py_ssize_t i = 0; !need && i < n; i++) need = order[index[item(f.inputs, i)]].need;
        index[f.v] = (int)order.size();
        order.push_back({f.v, f.inputs, f.rule, need, target});
        stack.pop_back();
    }
    std::vector<Ref> d(order.size());
    d[index[loss]] = Ref(Py_NewRef(dout0));
    auto add = [&](PyObject* inp, Ref g) -> bool {
        if (!g) return false;
        if (g.p == Py_None) return true;
        const int di = dtype_code(V(inp)->dtype);
        if (is_float(di) && dtype_code(V(g.p)->dtype) != di) g = Ref(cast_to(g.p, di));
        if (!g) return false;
        Ref& slot = d[index[inp]];
        if (slot) g = Ref(binary(slot.p, g.p, o_add));
        if (!g) return false;
        slot = std::move(g);
        return true;
    };
    for (size_t at = order.size(); at-- > 0;) {
        const Node& n = order[at];
        if (!n.need || n.target || !d[at] || !n.inputs) continue;
        const Py_ssize_t k = count(n.inputs);
        if (n.rule) {
            Ref want(PyList_New(k));
            if (!want) return nullptr;
            for (Py_ssize_t i = 0; i < k; i++) PyList_SET_ITEM(want.p, i, Py_NewRef(order[index[item(n.inputs, i)]].need ? Py_True : Py_False));
            Ref gs(PyObject_CallFunctionObjArgs(PyTuple_GET_ITEM(V(n.v)->vjp, 1), n.v, d[at].p, want.p, nullptr));
            if (!gs) return nullptr;
            Ref seq(PySequence_Fast(gs.p, "a gradient rule returns a sequence"));
            if (!seq) return nullptr;
            for (Py_ssize_t i = 0; i < k && i < PySequence_Fast_GET_SIZE(seq.p); i++)
                if (order[index[item(n.inputs, i)]].need && !add(item(n.inputs, i), Ref(Py_NewRef(PySequence_Fast_GET_ITEM(seq.p, i))))) return nullptr;
        } else
            for (Py_ssize_t i = 0; i < k; i++)
                if (order[index[item(n.inputs, i)]].need && !add(item(n.inputs, i), Ref(op_grad(n.v, d[at].p, i)))) return nullptr;
    }
    PyObject* out = PyList_New(PyList_GET_SIZE(targets));
    for (Py_ssize_t i = 0; out && i < PyList_GET_SIZE(targets); i++) {
        auto it = index.find(PyList_GET_ITEM(targets, i));
        PyList_SET_ITEM(out, i, Py_NewRef(it != index.end() && d[it->second] ? d[it->second].p : Py_None));
    }
    return out;
}
PyObject* m_binary(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 3) { PyErr_SetString(PyExc_TypeError, "binary(x, y, op)"); return nullptr; }
    return binary(a[0], a[1], a[2]);
}
PyObject* m_unary(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "unary(x, op)"); return nullptr; }
    Ref op(PyUnicode_Check(a[1]) ? Py_NewRef(a[1]) : PyObject_Str(a[1]));
    return op ? unary(a[0], op.p) : nullptr;
}
PyObject* m_ternary(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 3) { PyErr_SetString(PyExc_TypeError, "ternary(cond, x, y)"); return nullptr; }
    return ternary(a[0], a[1], a[2]);
}
// reduce(x, op, dims, keepdims): a whole number or a sequence of them; () or None folds every axis
PyObject* m_reduce(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 4) { PyErr_SetString(PyExc_TypeError, "reduce(x, op, dims, keepdims)"); return nullptr; }
    Ref x(to_var(a[0]));
    if (!x) return nullptr;
    const Py_ssize_t nd = rank_of(x.p);
    long mask = 0;
    auto axis = [&](PyObject* d) {
        Ref i(PyNumber_Long(d));
        long v = i ? PyLong_AsLong(i.p) : -1;
        if (v == -1 && PyErr_Occurred()) return false;
        if (v < 0) v += nd;
        if (v < 0 || v >= nd) { PyErr_Format(PyExc_ValueError, "Wrong dims number: %R", a[2]); return false; }
        mask |= 1l << v;
        return true;
    };
    if (PyLong_Check(a[2])) { if (!axis(a[2])) return nullptr; }
    else if (a[2] != Py_None) {
        Ref seq(PySequence_Fast(a[2], "dims: a whole number or a sequence of them"));
        if (!seq) return nullptr;
        for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq.p); i++) if (!axis(PySequence_Fast_GET_ITEM(seq.p, i))) return nullptr;
    }
    if (!mask) mask = (1l << nd) - 1;
    const int keep = PyObject_IsTrue(a[3]);
    return keep < 0 ? nullptr : reduce(x.p, a[1], mask, keep ? (1l << nd) - 1 : 0);
}
PyObject* m_to_var(PyObject*, PyObject* x) { return to_var(x); }
// setup_graph(Var, dtypes, infer_binary, infer_unary, infer_reduce, to_var, op_grad)
PyObject* m_setup_graph(PyObject*, PyObject* args) {
    PyObject *var, *dtypes, *b, *u, *r, *tv, *og;
    if (!PyArg_ParseTuple(args, "OO!OOOOO", &var, &PyTuple_Type, &dtypes, &b, &u, &r, &tv, &og)) return nullptr;
    h_var_type = Py_NewRef(var);
    for (int i = 0; i < 10; i++) h_dtypes[i] = Py_NewRef(PyTuple_GET_ITEM(dtypes, i));
    h_infer_binary = Py_NewRef(b); h_infer_unary = Py_NewRef(u); h_infer_reduce = Py_NewRef(r); h_to_var = Py_NewRef(tv); h_op_grad = Py_NewRef(og);
    Py_RETURN_NONE;
}

// optim_step(kind, params, grads, states0, states1 or None, hyper, nesterov) -> False where a tensor is not float32 on the GPU.
// The new values of a step live in flat buffers per slot that hold up to kPackFloats elements of small parameters; the Vars are
// rebound to views of them. Whoever keeps one parameter of a step keeps its buffer: 1 MB at most, or a large parameter's own.
constexpr int64_t kPackFloats = 1 << 18;
decltype(&b200jt_optim_step) g_optim = nullptr;
PyObject* m_optim_step(PyObject*, PyObject* args) {
    const char* kind;
    PyObject *lists[4], *hyper;
    int nesterov;
    if (!PyArg_ParseTuple(args, "sO!O!O!OO!i", &kind, &PyList_Type, &lists[0], &PyList_Type, &lists[1], &PyList_Type, &lists[2], &lists[3], &PyTuple_Type,
                          &hyper, &nesterov)) return nullptr;
    const bool two = lists[3] != Py_None;
    const Py_ssize_t n = PyList_GET_SIZE(lists[0]);
    if (!g_optim || n == 0) Py_RETURN_FALSE;
    std::vector<const float*> in[4];
    std::vector<int64_t> sizes;
    for (int l = 0; l < (two ? 4 : 3); l++) {
        if (!PyList_Check(lists[l]) || PyList_GET_SIZE(lists[l]) != n) { PyErr_SetString(PyExc_ValueError, "optim_step: lists differ in length"); return nullptr; }
        for (Py_ssize_t i = 0; i < n; i++) {
            PyObject* v = PyList_GET_ITEM(lists[l], i);
            if (!is_var(v) || none(V(v)->data) || !THPVariable_Check(V(v)->data)) Py_RETURN_FALSE;
            const at::Tensor& t = THPVariable_Unpack(V(v)->data);
            if (!t.is_cuda() || !t.is_contiguous() || t.scalar_type() != at::kFloat || (l && t.numel() != sizes[i])) Py_RETURN_FALSE;
            if (l == 0) sizes.push_back(t.numel());
            in[l].push_back((const float*)t.const_data_ptr());
        }
    }
    std::vector<double> h;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(hyper); i++) h.push_back(PyFloat_AsDouble(PyTuple_GET_ITEM(hyper, i)));
    if (PyErr_Occurred()) return nullptr;
    HANDLE_TH_ERRORS
    {
        const auto device = c10::Device(c10::kCUDA, c10::cuda::current_device());
        static const int slot[3] = {0, 2, 3};
        std::vector<int64_t> total;                                        // of each buffer
        std::vector<std::pair<size_t, int64_t>> place;                     // of each parameter: (buffer, offset)
        for (int64_t s : sizes) {
            const int64_t room = (s + 3) / 4 * 4;
            if (total.empty() || total.back() + room > kPackFloats) total.push_back(0);
            place.emplace_back(total.size() - 1, total.back());
            total.back() += room;
        }
        std::vector<at::Tensor> flat[3];
        std::vector<float*> out[3];
        for (int o = 0; o < (two ? 3 : 2); o++) {
            for (int64_t t : total) flat[o].push_back(at::Tensor(at::detail::empty_cuda({t}, at::kFloat, device, std::nullopt)));
            for (auto& p : place) out[o].push_back((float*)flat[o][p.first].data_ptr() + p.second);
        }
        const int rc = g_optim(kind, (int)n, sizes.data(), in[0].data(), in[1].data(), in[2].data(), two ? in[3].data() : nullptr, out[0].data(), out[1].data(),
                               two ? out[2].data() : nullptr, h.data(), (int)h.size(), nesterov, (void*)c10::cuda::getCurrentCUDAStream().stream());
        if (rc) { PyErr_Format(h_error, "optim_step: %s (status %d)", g_last_error ? g_last_error() : "", rc); return nullptr; }
        for (int o = 0; o < (two ? 3 : 2); o++) {
            for (Py_ssize_t i = 0; i < n; i++) {
                VarObj* v = V(PyList_GET_ITEM(lists[slot[o]], i));
                const at::Tensor& old = THPVariable_Unpack(v->data);
                PyObject* py = THPVariable_Wrap(flat[o][place[i].first].as_strided(old.sizes(), old.strides(), place[i].second));
                if (!py) return nullptr;
                Py_XSETREF(v->data, py);
                // as Var.assign: nothing describes the value it held before
                Py_CLEAR(v->builder); Py_CLEAR(v->relay); Py_CLEAR(v->vjp); Py_CLEAR(v->bn_running); Py_CLEAR(v->konst);
                Py_XSETREF(v->op, Py_NewRef(Py_None));
            }
        }
    }
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------------ module functions
// realize(roots) -> True when every root is computed; False: the caller has to run the Python planner.
PyObject* m_realize(PyObject* self, PyObject* arg) {
    PyObject* seq = PySequence_Fast(arg, "realize: a list of Vars");
    if (!seq) return nullptr;
    struct Hold { PyObject* o; ~Hold() { Py_DECREF(o); } } hold{seq};
    std::vector<VarObj*> roots;
    for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); i++) {
        PyObject* o = PySequence_Fast_GET_ITEM(seq, i);
        if (!is_var(o)) Py_RETURN_FALSE;
        if (none(((VarObj*)o)->data)) roots.push_back((VarObj*)o);
    }
    if (roots.empty()) Py_RETURN_TRUE;
    if (g_recording || !h_record) Py_RETURN_FALSE;
    HANDLE_TH_ERRORS                                        // torch's own errors: running out of memory is torch.OutOfMemoryError, as in the planner
    {
        Walk w;
        w.run(roots);
        if (!w.ok) Py_RETURN_FALSE;
        bool waited = false;
        for (VarObj* v : w.leaves)
            if (!none(v->pending)) {                        // produced by a collective on another stream
                PyObject* r = PyObject_CallMethodNoArgs((PyObject*)v, s_wait);
                if (!r) return nullptr;
                Py_DECREF(r);
                waited = true;
            }
        if (waited) return m_realize(self, arg);            // other threads ran: the graph is looked at again
        if (const std::shared_ptr<Tape>* found = find_tape(w.key)) {
            const std::shared_ptr<Tape> tape = *found;
            if (!tape) Py_RETURN_FALSE;
            if (!replay(*tape, w)) return nullptr;
            Py_RETURN_TRUE;
        }
        if (!w.numbers.empty() && ++g_variants[w.skeleton()] > kMaxVariants) Py_RETURN_FALSE;
        PyObject* nodes = PyList_New((Py_ssize_t)w.nodes.size());
        PyObject* leaves = PyList_New((Py_ssize_t)w.leaves.size());
        for (size_t i = 0; i < w.nodes.size(); i++) PyList_SET_ITEM(nodes, (Py_ssize_t)i, Py_NewRef((PyObject*)w.nodes[i]));
        for (size_t i = 0; i < w.leaves.size(); i++) PyList_SET_ITEM(leaves, (Py_ssize_t)i, Py_NewRef((PyObject*)w.leaves[i]));
        g_recording = true;
        PyObject* spec = PyObject_CallFunctionObjArgs(h_record, seq, nodes, leaves, nullptr);
        g_recording = false;
        Py_DECREF(nodes);
        Py_DECREF(leaves);
        if (!spec) return nullptr;
        age_tapes();
        std::shared_ptr<Tape> tape;
        if (spec != Py_None) {
            tape = build_tape(spec, (int)w.leaves.size());
            if (!tape) { Py_DECREF(spec); if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "tape: malformed record"); return nullptr; }
            g_records++;
        }
        g_tapes.emplace(std::move(w.key), std::move(tape));
        Py_DECREF(spec);
        Py_RETURN_TRUE;
    }
    END_HANDLE_TH_ERRORS
}

// setup(Shape, make_shape, DType, canon, record, error, flags dict, {symbol: address})
PyObject* m_setup(PyObject*, PyObject* args) {
    PyObject *shape, *make, *dtype, *canon, *record, *error, *flags, *symbols;
    if (!PyArg_ParseTuple(args, "OOOOOOO!O!", &shape, &make, &dtype, &canon, &record, &error, &PyDict_Type, &flags, &PyDict_Type, &symbols))
        return nullptr;
    h_shape_type = Py_NewRef(shape); h_make_shape = Py_NewRef(make); h_dtype_type = Py_NewRef(dtype); h_canon = Py_NewRef(canon);
    h_record = record == Py_None ? nullptr : Py_NewRef(record);
    h_error = Py_NewRef(error); h_flags = Py_NewRef(flags);
    for (Entry& e : g_entries)
        if (PyObject* a = PyDict_GetItemString(symbols, e.name)) e.fn = PyLong_AsVoidPtr(a);
    if (PyObject* a = PyDict_GetItemString(symbols, "b200jt_last_error")) g_last_error = (const char* (*)())PyLong_AsVoidPtr(a);
    if (PyObject* a = PyDict_GetItemString(symbols, "b200jt_optim_step")) g_optim = (decltype(g_optim))PyLong_AsVoidPtr(a);
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}
PyObject* m_set_record(PyObject*, PyObject* f) {
    Py_XSETREF(h_record, Py_NewRef(f));
    Py_RETURN_NONE;
}
PyObject* m_context(PyObject*, PyObject* n) {
    g_context = PyLong_AsLong(n);
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}
PyObject* m_clear(PyObject*, PyObject*) { g_tapes.clear(); g_older.clear(); g_variants.clear(); Py_RETURN_NONE; }
PyObject* m_stats(PyObject*, PyObject*) {
    return Py_BuildValue("{s:n,s:L,s:L}", "tapes", (Py_ssize_t)(g_tapes.size() + g_older.size()), "recorded", (long long)g_records, "replayed", (long long)g_replays);
}
PyObject* m_take_plans(PyObject*, PyObject*) {
    const long long n = g_plans;
    g_plans = 0;
    return PyLong_FromLongLong(n);
}
PyMethodDef methods[] = {
    {"binary", (PyCFunction)(void*)m_binary, METH_FASTCALL, nullptr}, {"unary", (PyCFunction)(void*)m_unary, METH_FASTCALL, nullptr},
    {"ternary", (PyCFunction)(void*)m_ternary, METH_FASTCALL, nullptr}, {"reduce", (PyCFunction)(void*)m_reduce, METH_FASTCALL, nullptr},
    {"to_var", m_to_var, METH_O, nullptr}, {"backprop", m_backprop, METH_VARARGS, nullptr}, {"setup_graph", m_setup_graph, METH_VARARGS, nullptr},
    {"optim_step", m_optim_step, METH_VARARGS, nullptr},
    {"realize", m_realize, METH_O, nullptr}, {"setup", m_setup, METH_VARARGS, nullptr}, {"set_record", m_set_record, METH_O, nullptr},
    {"set_context", m_context, METH_O, nullptr}, {"clear", m_clear, METH_NOARGS, nullptr}, {"stats", m_stats, METH_NOARGS, nullptr},
    {"take_plans", m_take_plans, METH_NOARGS, nullptr}, {nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200jt_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__b200jt_host(void) {
    OpType.tp_name = "_b200jt_host.Op";
    OpType.tp_basicsize = sizeof(OpObj);
    OpType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
    OpType.tp_new = PyType_GenericNew;
    OpType.tp_init = (initproc)op_init;
    OpType.tp_traverse = (traverseproc)op_traverse;
    OpType.tp_clear = (inquiry)op_clear;
    OpType.tp_dealloc = (destructor)op_dealloc;
    OpType.tp_members = op_members;
    VarType.tp_name = "_b200jt_host.VarBase";
    VarType.tp_basicsize = sizeof(VarObj);
    VarType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC;
    VarType.tp_new = PyType_GenericNew;
    VarType.tp_init = (initproc)var_init;
    VarType.tp_traverse = (traverseproc)var_traverse;
    VarType.tp_clear = (inquiry)var_clear;
    VarType.tp_dealloc = (destructor)var_dealloc;
    VarType.tp_members = var_members;
    VarType.tp_getset = var_getset;
    if (PyType_Ready(&OpType) < 0 || PyType_Ready(&VarType) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module);
    if (!m) return nullptr;
    s_running_mean = PyUnicode_InternFromString("running_mean"); s_running_var = PyUnicode_InternFromString("running_var");
    s_momentum = PyUnicode_InternFromString("momentum"); s_wait = PyUnicode_InternFromString("wait");
    s_sig = PyUnicode_InternFromString("sig"); s_also = PyUnicode_InternFromString("also");
    s_custom = PyUnicode_InternFromString("custom"); s_fuse = PyUnicode_InternFromString("b200_fuse_chains");
    struct { PyObject** at; const char* text; } names[] = {
        {&k_binary, "binary"}, {&k_unary, "unary"}, {&k_ternary, "ternary"}, {&k_reduce, "reduce"}, {&k_fill, "fill"}, {&k_broadcast, "broadcast_to"},
        {&k_reshape, "reshape"}, {&k_reindex, "reindex"}, {&k_op, "op"}, {&k_value, "value"}, {&k_mask, "bcast_mask"}, {&k_keep, "keepdims_mask"},
        {&k_rmask, "reduce_mask"}, {&s_amp, "amp_reg"}, {&o_add, "add"}, {&o_subtract, "subtract"}, {&o_multiply, "multiply"}, {&o_divide, "divide"},
        {&o_maximum, "maximum"}, {&o_minimum, "minimum"}, {&o_equal, "equal"}, {&o_negative, "negative"}, {&o_mean, "mean"}, {&o_log, "log"}, {&o_exp, "exp"}};
    for (auto& n : names) *n.at = PyUnicode_InternFromString(n.text);
    i_zero = PyLong_FromLong(0);
    s_collective = PyUnicode_InternFromString("mpi_all_reduce"); s_value = PyUnicode_InternFromString("value");
    s_wgrad = PyUnicode_InternFromString("b200_wgrad_tc");
    if (PyModule_AddObjectRef(m, "Op", (PyObject*)&OpType) < 0 || PyModule_AddObjectRef(m, "VarBase", (PyObject*)&VarType) < 0) return nullptr;
    return m;
}
