// The entry points that a program calls thousands of times a second, as functions of a CPython module: the Python mirror
// (ferrograd_b200/backend.py, graph.py) goes through it where a foreign-function call's argument conversion (2.5 us, and twice that
// for an elementwise program) takes as long as a small kernel.  Same C ABI, same status codes; a call takes 0.3 us.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/ferrograd_b200.h"

namespace {

bool take_integer(PyObject* o, unsigned long long* out) {
    if (PyLong_CheckExact(o)) {
        *out = PyLong_AsUnsignedLongLongMask(o);
        return !PyErr_Occurred();
    }
    PyObject* const i = PyNumber_Index(o);
    if (!i) return false;
    *out = PyLong_AsUnsignedLongLongMask(i);
    Py_DECREF(i);
    return !PyErr_Occurred();
}
// A device pointer or a handle: None, an address, something with an address in `ptr` (a tensor, a buffer), or a ctypes c_void_p.
bool take_address(PyObject* o, void** out) {
    *out = nullptr;
    if (o == Py_None) return true;
    if (PyLong_CheckExact(o)) {
        *out = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(o);
        return !PyErr_Occurred();
    }
    const bool handle = strcmp(Py_TYPE(o)->tp_name, "c_void_p") == 0;
    PyObject* a = PyObject_GetAttrString(o, handle ? "value" : "ptr");
    if (!a && !handle && PyErr_ExceptionMatches(PyExc_AttributeError)) {
        PyErr_Clear();
        a = PyNumber_Long(o);
    }
    if (!a) return false;
    if (a != Py_None) *out = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(a);
    Py_DECREF(a);
    return !PyErr_Occurred();
}
template <typename T>
bool take(PyObject* o, T* out) {
    if constexpr (std::is_pointer_v<T>) {
        void* p;
        if (!take_address(o, &p)) return false;
        *out = static_cast<T>(p);
        return true;
    } else if constexpr (std::is_floating_point_v<T>) {
        const double v = PyFloat_AsDouble(o);
        *out = (T)v;
        return v != -1.0 || !PyErr_Occurred();
    } else {
        unsigned long long v = 0;
        if (!take_integer(o, &v)) return false;
        *out = (T)v;
        return true;
    }
}

template <typename... A, size_t... I>
PyObject* invoke(int32_t (*f)(A...), PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<A...> v;
    if (!(take(args[I], &std::get<I>(v)) && ...)) return nullptr;
    int32_t code;
    Py_BEGIN_ALLOW_THREADS
    code = f(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}
template <typename... A>
PyObject* call(int32_t (*f)(A...), PyObject* const* args, Py_ssize_t n) {
    if (n != (Py_ssize_t)sizeof...(A)) {
        PyErr_Format(PyExc_TypeError, "%d arguments expected, %zd given", (int)sizeof...(A), n);
        return nullptr;
    }
    return invoke(f, args, std::index_sequence_for<A...>{});
}
template <auto F>
PyObject* method(PyObject*, PyObject* const* args, Py_ssize_t n) { return call(F, args, n); }

// ---- elementwise programs: a sequence of (op, a, b, imm), op a number or a name ----
PyObject* op_numbers = nullptr;      // name -> number
struct Array {      // a small array that goes with the scope
    void* p;
    explicit Array(size_t bytes) : p(PyMem_Malloc(bytes ? bytes : 1)) { if (!p) PyErr_NoMemory(); }
    ~Array() { PyMem_Free(p); }
    Array(const Array&) = delete;
    Array& operator=(const Array&) = delete;
};
struct Sequence {
    PyObject* o;
    Sequence(PyObject* x, const char* what) : o(PySequence_Fast(x, what)) {}
    ~Sequence() { Py_XDECREF(o); }
    Sequence(const Sequence&) = delete;
    Sequence& operator=(const Sequence&) = delete;
    Py_ssize_t size() const { return PySequence_Fast_GET_SIZE(o); }
    PyObject* at(Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(o, i); }
};
bool take_program(const Sequence& s, fg_ew_instr* out) {
    for (Py_ssize_t i = 0; i < s.size(); ++i) {
        Sequence t(s.at(i), "an instruction is (op, a, b, imm)");
        if (!t.o) return false;
        if (t.size() != 4) {
            PyErr_SetString(PyExc_ValueError, "an instruction is (op, a, b, imm)");
            return false;
        }
        PyObject* op = t.at(0);
        if (PyUnicode_Check(op)) {
            PyObject* const number = PyDict_GetItemWithError(op_numbers, op);
            if (!number) {
                if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, op);
                return false;
            }
            op = number;
        }
        if (!take(op, &out[i].op) || !take(t.at(1), &out[i].a) || !take(t.at(2), &out[i].b) || !take(t.at(3), &out[i].imm)) return false;
    }
    return true;
}
bool take_addresses(const Sequence& s, void** out) {
    for (Py_ssize_t i = 0; i < s.size(); ++i)
        if (!take_address(s.at(i), &out[i])) return false;
    return true;
}
// chain_fwd(ctx, dtype, n, program, inputs, out, saved): saved is None or an address (or None) for each instruction.
PyObject* chain_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    fg_ctx* ctx;
    int32_t dtype, code;
    uint64_t count;
    void* out;
    if (n != 7) { PyErr_SetString(PyExc_TypeError, "chain_fwd: 7 arguments expected"); return nullptr; }
    if (!take(a[0], &ctx) || !take(a[1], &dtype) || !take(a[2], &count) || !take_address(a[5], &out)) return nullptr;
    Sequence program(a[3], "the program is a sequence"), inputs(a[4], "the inputs are a sequence");
    if (!program.o || !inputs.o) return nullptr;
    Sequence saved(a[6] == Py_None ? a[3] : a[6], "saved is a sequence");
    if (!saved.o) return nullptr;
    Array prog(program.size() * sizeof(fg_ew_instr)), in(inputs.size() * sizeof(void*)), keep(program.size() * sizeof(void*));
    if (!prog.p || !in.p || !keep.p || !take_program(program, (fg_ew_instr*)prog.p) || !take_addresses(inputs, (void**)in.p)) return nullptr;
    if (a[6] != Py_None) {
        if (saved.size() != program.size()) { PyErr_SetString(PyExc_ValueError, "one saved address for each instruction"); return nullptr; }
        if (!take_addresses(saved, (void**)keep.p)) return nullptr;
    }
    void* const* const kept = a[6] != Py_None ? (void* const*)keep.p : nullptr;
    Py_BEGIN_ALLOW_THREADS
    code = fg_eltwise_chain_fwd_dt(ctx, dtype, count, (const fg_ew_instr*)prog.p, (int32_t)program.size(), (const void* const*)in.p,
                                   (int32_t)inputs.size(), out, kept);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}
// chain_bwd(ctx, dtype, n, program, inputs, seed, grads, accumulate)
PyObject* chain_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    fg_ctx* ctx;
    int32_t dtype, accumulate, code;
    uint64_t count;
    void* seed;
    if (n != 8) { PyErr_SetString(PyExc_TypeError, "chain_bwd: 8 arguments expected"); return nullptr; }
    if (!take(a[0], &ctx) || !take(a[1], &dtype) || !take(a[2], &count) || !take_address(a[5], &seed) || !take(a[7], &accumulate)) return nullptr;
    Sequence program(a[3], "the program is a sequence"), inputs(a[4], "the inputs are a sequence"), grads(a[6], "the gradients are a sequence");
    if (!program.o || !inputs.o || !grads.o) return nullptr;
    if (grads.size() > inputs.size()) { PyErr_SetString(PyExc_IndexError, "more gradients than inputs"); return nullptr; }
    Array prog(program.size() * sizeof(fg_ew_instr)), in(inputs.size() * sizeof(void*)), out(inputs.size() * sizeof(void*));
    if (!prog.p || !in.p || !out.p) return nullptr;
    memset(out.p, 0, inputs.size() * sizeof(void*));      // inputs without a gradient
    if (!take_program(program, (fg_ew_instr*)prog.p) || !take_addresses(inputs, (void**)in.p) || !take_addresses(grads, (void**)out.p)) return nullptr;
    Py_BEGIN_ALLOW_THREADS
    code = fg_eltwise_chain_bwd_dt(ctx, dtype, count, (const fg_ew_instr*)prog.p, (int32_t)program.size(), (const void* const*)in.p,
                                   (int32_t)inputs.size(), seed, (void* const*)out.p, accumulate);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

#define FG_METHOD(name) {#name, (PyCFunction)(void (*)(void))method<name>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FG_METHOD(fg_gemm_f32), FG_METHOD(fg_gemm_bwd_f32), FG_METHOD(fg_gemm_paired_f32), FG_METHOD(fg_gemm_bwd_paired_f32),
    FG_METHOD(fg_gemm_batched_f32), FG_METHOD(fg_gemm_batched_bwd_f32), FG_METHOD(fg_gemm_lowp), FG_METHOD(fg_gemm_bwd_lowp),
    FG_METHOD(fg_bias_act_fwd), FG_METHOD(fg_act_bwd), FG_METHOD(fg_softmax_fwd), FG_METHOD(fg_softmax_bwd),
    FG_METHOD(fg_softmax_ce_fwd_bwd), FG_METHOD(fg_ce_loss_grad), FG_METHOD(fg_mse_loss_grad), FG_METHOD(fg_bce_loss_grad),
    FG_METHOD(fg_sgd_step), FG_METHOD(fg_convert), FG_METHOD(fg_plan_launch),
    FG_METHOD(fg_exec_dispatch_forward), FG_METHOD(fg_exec_dispatch_loss), FG_METHOD(fg_exec_dispatch_backward), FG_METHOD(fg_exec_dispatch_optim),
    {"chain_fwd", (PyCFunction)(void (*)(void))chain_fwd, METH_FASTCALL, nullptr},
    {"chain_bwd", (PyCFunction)(void (*)(void))chain_bwd, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef definition = {PyModuleDef_HEAD_INIT, "_calls", "Entry points of libferrograd_b200.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) {
    static const char* const names[] = {"input", "const", "add", "sub", "mul", "div", "neg", "abs", "exp", "log", "tanh", "relu", "gelu", "elu"};
    PyObject* const m = PyModule_Create(&definition);
    if (!m) return nullptr;
    op_numbers = PyDict_New();
    for (long i = 0; op_numbers && i < (long)(sizeof(names) / sizeof(names[0])); ++i) {
        PyObject* const v = PyLong_FromLong(i);
        if (!v || PyDict_SetItemString(op_numbers, names[i], v) != 0) { Py_XDECREF(v); Py_CLEAR(op_numbers); break; }
        Py_DECREF(v);
    }
    if (!op_numbers || PyModule_AddObjectRef(m, "OPS", op_numbers) != 0) { Py_DECREF(m); return nullptr; }
    return m;
}
