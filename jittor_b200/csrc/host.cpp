// Native host path: the Var / Op objects of the lazy graph and the replay of planned graphs.
//
// What bounded it before: a graph was matched, fused and launched by Python on every sync -- 0.1 ms for a softmax and its
// gradient, 3 ms for a convolution + BatchNorm + ReLU block with its gradients, whose kernels take 0.35 ms. A program runs the
// same few graphs over and over with other tensors, so the first sync of a graph runs the Python planner with every
// allocation and library call written to a tape (executor.py), and later syncs of a graph of the same structure replay that
// tape from here: one walk over the graph makes its signature (op kinds, attributes, shapes, dtypes, how nodes share
// inputs, alignment of the leaves), a hash lookup finds the tape, and its calls run with the new pointers. Results are not
// kept: every replay allocates its outputs and launches every kernel again.
#include <Python.h>
#include <structmember.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

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
PyObject *s_running_mean, *s_running_var, *s_momentum, *s_wait, *s_sig, *s_also, *s_custom, *s_fuse, *s_wgrad, *s_collective;
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

int var_init(VarObj* self, PyObject* args, PyObject* kw) {
    static const char* names[] = {"shape", "dtype", "op", "data", "is_scalar", nullptr};
    PyObject *shape, *dtype, *op = Py_None, *data = Py_None;
    int scalar = 0;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "OO|OOp", (char**)names, &shape, &dtype, &op, &data, &scalar)) return -1;
    if ((PyObject*)Py_TYPE(shape) == h_shape_type) Py_INCREF(shape);
    else if (!(shape = PyObject_CallOneArg(h_make_shape, shape))) return -1;
    if ((PyObject*)Py_TYPE(dtype) == h_dtype_type) Py_INCREF(dtype);
    else if (!(dtype = PyObject_CallOneArg(h_canon, dtype))) { Py_DECREF(shape); return -1; }
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
        Py_DECREF(b);
        if (!op) return nullptr;
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
    std::unordered_map<const void*, int> index;      // Var -> number: leaves and nodes share one numbering in visiting order
    bool ok = true;
    int count = 0;

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
    void meta(VarObj* v) {
        PyObject* s = v->shape;
        if (!s || !PyList_Check(s)) { ok = false; return; }
        const Py_ssize_t n = PyList_GET_SIZE(s);
        tag((char)('A' + n));
        for (Py_ssize_t i = 0; i < n; i++) num(PyLong_AsLongLong(PyList_GET_ITEM(s, i)));
        text(v->dtype);
        if (!none(v->konst)) { tag('c'); value(v->konst); }
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
                while (PyDict_Next(o->attrs, &pos, &k, &x)) { text(k); value(x); }
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
    void run(const std::vector<VarObj*>& roots) {
        key.reserve(2048);
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
                if (f.next == 0 && f.kids.empty() && none(f.v->data)) children(f.v, f.kids);
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
    E(b200jt_softmax), E(b200jt_softmax_backward), E(b200jt_layer_norm), E(b200jt_matmul_workspace), E(b200jt_matmul),
    E(b200jt_batched_matmul), E(b200jt_conv2d_workspace), E(b200jt_conv2d), E(b200jt_conv2d_formats_workspace), E(b200jt_conv2d_formats),
    E(b200jt_conv2d_transpose), E(b200jt_conv2d_backward_w), E(b200jt_conv2d_backward_w_workspace), E(b200jt_conv2d_backward_w_tc),
    E(b200jt_conv2d_backward_w_formats_workspace), E(b200jt_conv2d_backward_w_formats), E(b200jt_bn_stats), E(b200jt_bn_apply),
    E(b200jt_layer_norm_backward_workspace), E(b200jt_layer_norm_backward), E(b200jt_bn_backward_sums),
    E(b200jt_bn_backward_dx), E(b200jt_pool2d), E(b200jt_pool2d_backward), E(b200jt_pool2d_backward_indices),
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
    std::vector<Slot> slots;
    std::vector<Patch> patches;
    std::vector<std::pair<int, int>> nbytes;   // (slot, buffer): the size of a workspace passed beside its pointer
    int stream = -1;                       // slot of the stream
    std::vector<int> release;              // buffers nothing reads after this step
};
struct Result { int node, buf; bool same; int64_t off; std::vector<int64_t> shape; };
struct Tape {
    int n_leaves = 0, n_bufs = 0, n_plans = 0;
    std::vector<Step> steps;
    std::vector<Result> results;
    std::vector<int> bn_done;              // nodes whose running statistics the fused BatchNorm updated
    // storage behind the slots
    std::deque<std::vector<b200jt_tensor>> tensors;
    std::deque<std::string> strings;
    std::deque<std::vector<const char*>> string_lists;
    std::deque<std::vector<int64_t>> longs;
    std::deque<std::vector<int32_t>> ints;
    std::vector<at::Tensor> bufs;
};
std::unordered_map<std::string, std::unique_ptr<Tape>> g_tapes;      // null: the planner has to run every time

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

// spec: (number of buffers, steps, results, nodes whose running statistics moved, plans) from executor._record
std::unique_ptr<Tape> build_tape(PyObject* spec, int n_leaves) {
    PyObject *steps, *results, *bn;
    auto t = std::make_unique<Tape>();
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
            PyObject* args = PyTuple_GET_ITEM(s, 3);
            st.slots.reserve((size_t)PyList_GET_SIZE(args));
            for (Py_ssize_t k = 0; k < PyList_GET_SIZE(args); k++) if (!add_arg(*t, st, PyList_GET_ITEM(args, k))) return nullptr;
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
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(bn); i++) t->bn_done.push_back((int)PyLong_AsLong(PyList_GET_ITEM(bn, i)));
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

bool replay(Tape& t, const Walk& w) {
    t.bufs.assign((size_t)t.n_bufs, at::Tensor());
    struct Clear { Tape& t; ~Clear() { t.bufs.clear(); } } clear{t};
    for (int i = 0; i < t.n_leaves; i++) {
        VarObj* v = w.leaves[i];
        if (!none(v->pending)) {                           // produced by a collective on another stream
            PyObject* r = PyObject_CallMethodNoArgs((PyObject*)v, s_wait);
            if (!r) return false;
            Py_DECREF(r);
        }
        t.bufs[i] = THPVariable_Unpack(v->data);
    }
    const auto device = c10::Device(c10::kCUDA, c10::cuda::current_device());
    void* stream = (void*)c10::cuda::getCurrentCUDAStream().stream();
    for (Step& st : t.steps) {
        if (st.kind == Step::ALLOC) {
            t.bufs[st.buf] = at::Tensor(at::detail::empty_cuda(st.sizes, st.type, device, std::nullopt));
            continue;
        }
        if (st.kind == Step::FILL) { t.bufs[st.buf].fill_(st.value); continue; }
        for (Patch& p : st.patches) {
            const at::Tensor& b = t.bufs[p.buf];
            *p.where = b.defined() ? (char*)b.data_ptr() + p.off : nullptr;
        }
        for (auto& n : st.nbytes) st.slots[n.first].i = t.bufs[n.second].defined() ? t.bufs[n.second].numel() : 0;
        if (st.stream >= 0) st.slots[st.stream].p = stream;
        const int64_t rc = st.entry->invoke(st.entry->fn, st.slots.data());
        if (st.kind == Step::WORKSPACE) {
            if (rc > 0) t.bufs[st.buf] = at::Tensor(at::detail::empty_cuda({rc}, at::kByte, device, std::nullopt));
        } else if (rc != 0) {
            PyErr_Format(h_error, "%s: %s (status %d)", st.entry->name + 7, g_last_error ? g_last_error() : "", (int)rc);
            return false;
        }
        for (int b : st.release) t.bufs[b].reset();
    }
    for (const Result& r : t.results) {
        at::Tensor out = t.bufs[r.buf];
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
    for (int n : t.bn_done) Py_XSETREF(w.nodes[n]->bn_running, Py_NewRef(Py_None));
    g_plans += t.n_plans;
    g_replays++;
    return true;
}

// ------------------------------------------------------------------------------------------------ module functions
// realize(roots) -> True when every root is computed; False: the caller has to run the Python planner.
PyObject* m_realize(PyObject*, PyObject* arg) {
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
    Walk w;
    try {
        w.run(roots);
        if (!w.ok) Py_RETURN_FALSE;
        auto it = g_tapes.find(w.key);
        if (it != g_tapes.end()) {
            if (!it->second) Py_RETURN_FALSE;
            if (!replay(*it->second, w)) return nullptr;
            Py_RETURN_TRUE;
        }
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
        if (g_tapes.size() >= 4096) g_tapes.clear();          // programs with endless shapes: start over rather than grow
        std::unique_ptr<Tape> tape;
        if (spec != Py_None) {
            tape = build_tape(spec, (int)w.leaves.size());
            if (!tape) { Py_DECREF(spec); if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "tape: malformed record"); return nullptr; }
            g_records++;
        }
        g_tapes.emplace(std::move(w.key), std::move(tape));
        Py_DECREF(spec);
        Py_RETURN_TRUE;
    } catch (const std::exception& e) {
        g_recording = false;
        PyErr_SetString(h_error ? h_error : PyExc_RuntimeError, e.what());
        return nullptr;
    }
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
PyObject* m_clear(PyObject*, PyObject*) { g_tapes.clear(); Py_RETURN_NONE; }
PyObject* m_stats(PyObject*, PyObject*) {
    return Py_BuildValue("{s:n,s:L,s:L}", "tapes", (Py_ssize_t)g_tapes.size(), "recorded", (long long)g_records, "replayed", (long long)g_replays);
}
PyObject* m_take_plans(PyObject*, PyObject*) {
    const long long n = g_plans;
    g_plans = 0;
    return PyLong_FromLongLong(n);
}
PyMethodDef methods[] = {
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
    s_collective = PyUnicode_InternFromString("mpi_all_reduce");
    s_wgrad = PyUnicode_InternFromString("b200_wgrad_tc");
    if (PyModule_AddObjectRef(m, "Op", (PyObject*)&OpType) < 0 || PyModule_AddObjectRef(m, "VarBase", (PyObject*)&VarType) < 0) return nullptr;
    return m;
}
