// The collective calls of the Python communicator as one native function call each.
//
// A call on eight ranks looks at sixteen tensors (type, place, layout, length, address) and eight
// streams. Through Python attributes and ctypes a 4 KiB call took 40 us of host time, over ten times what
// its kernel takes; with these checks native and one completion event instead of eight it takes 3.3 us
// (one rank, 8 KiB: 9.4 -> 2.9 us). The module knows the C interface only by two addresses handed over in
// bind(), so whichever build of the library the process loaded is the one that runs.
//
// The reference library (nano-nccl) has no Python layer; its C++ calls
// (include/nano_nccl/communicator.h:31-58) are what these methods forward to.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include "b200ccl/types.h"

#include <cstdint>
#include <exception>

namespace {

using CollectiveFn = int (*)(void*, int, const void* const*, void* const*, void* const*, std::size_t, int, int, int);
using LastErrorFn = const char* (*)();

CollectiveFn g_collective = nullptr;
LastErrorFn g_last_error = nullptr;
PyObject* g_error_class = nullptr;  // what a failed call raises; rejected arguments raise ValueError

constexpr int kMaxRanks = b200ccl::kMaxRanks;
constexpr const char* kOps[] = {"sum", "avg", "max", "min"};  // in the order of the C interface

// One communicator as its calls need it.
struct Caller {
    PyObject_HEAD
    void* handle;
    int local_ranks;
    long long world;
    int device[kMaxRanks];
};

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return 0;
        case at::kHalf: return 1;
        case at::kBFloat16: return 2;
        default: return -1;
    }
}

int op_code(PyObject* op) {
    if (PyUnicode_Check(op)) {
        for (int i = 0; i < 4; ++i)
            if (PyUnicode_CompareWithASCIIString(op, kOps[i]) == 0) return i;
    }
    PyErr_Format(PyExc_ValueError, "unknown reduction '%S'", op);
    return -1;
}

// The tensors of one side: one tensor, or a sequence with one per local rank. Borrowed from `held`.
struct Side {
    PyObject* held = nullptr;
    PyObject* item[kMaxRanks] = {nullptr};
    Py_ssize_t size = 0;
    bool single = false;
    ~Side() { Py_XDECREF(held); }

    bool read(PyObject* obj) {
        // (Whether a list is a tensor is asked of the tensor class, which takes as long as looking at five tensors.)
        if (!PyList_CheckExact(obj) && !PyTuple_CheckExact(obj) && THPVariable_Check(obj)) {
            single = true;
            size = 1;
            item[0] = obj;
            return true;
        }
        held = PySequence_Fast(obj, "collectives take a tensor, or a sequence with one tensor per local rank");
        if (held == nullptr) return false;
        size = PySequence_Fast_GET_SIZE(held);
        for (Py_ssize_t i = 0; i < size && i < kMaxRanks; ++i) item[i] = PySequence_Fast_GET_ITEM(held, i);
        return true;
    }
};

// Everything the C layer cannot see behind a raw pointer: a tensor that is too small, of another
// dtype or on another GPU would make the kernel write outside the allocation.
bool check_tensor(const char* what, int i, PyObject* obj, at::ScalarType dtype, std::int64_t numel, int device) {
    const bool is_tensor = THPVariable_Check(obj);
    if (!is_tensor || !THPVariable_Unpack(obj).is_cuda() || !THPVariable_Unpack(obj).is_contiguous()) {
        PyErr_Format(PyExc_ValueError, "%s[%d] must be a contiguous CUDA tensor", what, i);
        return false;
    }
    const at::Tensor& t = THPVariable_Unpack(obj);
    if (t.scalar_type() != dtype) {
        PyErr_Format(PyExc_ValueError, "%s[%d] has dtype %s, expected %s", what, i, c10::toString(t.scalar_type()), c10::toString(dtype));
        return false;
    }
    if (t.numel() != numel) {
        PyErr_Format(PyExc_ValueError, "%s[%d] has %lld elements, expected %lld", what, i, static_cast<long long>(t.numel()),
                     static_cast<long long>(numel));
        return false;
    }
    if (t.get_device() != device) {
        PyErr_Format(PyExc_ValueError, "%s[%d] lives on cuda:%d, local rank %d of this communicator drives cuda:%d", what, i,
                     static_cast<int>(t.get_device()), i, device);
        return false;
    }
    return true;
}

// A torch stream (anything with a cuda_stream attribute) or a raw handle as an integer.
bool stream_handle(PyObject* obj, void** out) {
    PyObject* attr = PyObject_GetAttrString(obj, "cuda_stream");
    if (attr == nullptr) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return false;
        PyErr_Clear();
        attr = PyNumber_Long(obj);
        if (attr == nullptr) return false;
    }
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(attr);
    Py_DECREF(attr);
    if (v == static_cast<unsigned long long>(-1) && PyErr_Occurred()) return false;
    *out = reinterpret_cast<void*>(static_cast<std::uintptr_t>(v));
    return true;
}

bool read_streams(const Caller* c, PyObject* streams, bool single, void** out) {
    const int n = c->local_ranks;
    if (streams == Py_None) {
        for (int i = 0; i < n; ++i) {
            out[i] = i > 0 && c->device[i] == c->device[0]
                         ? out[0]
                         : static_cast<void*>(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(c->device[i])).stream());
        }
        return true;
    }
    if (!PyList_Check(streams) && !PyTuple_Check(streams)) {
        if (!stream_handle(streams, &out[0])) return false;
        for (int i = 1; i < n; ++i) out[i] = out[0];
        return true;
    }
    const Py_ssize_t size = PySequence_Fast_GET_SIZE(streams);
    if (size < 1 || (!single && size != n)) {
        PyErr_Format(PyExc_ValueError, "need one stream per local rank (%d)", n);
        return false;
    }
    for (int i = 0; i < n; ++i)
        if (!stream_handle(PySequence_Fast_GET_ITEM(streams, i), &out[i])) return false;
    return true;
}

PyObject* run(Caller* c, int collective, PyObject* outs_obj, PyObject* inps_obj, PyObject* op_obj, PyObject* streams_obj) {
    if (c->handle == nullptr) {
        PyErr_SetString(PyExc_RuntimeError, "the communicator is closed");
        return nullptr;
    }
    Side outs, inps;
    if (!outs.read(outs_obj) || !inps.read(inps_obj)) return nullptr;
    const int n = c->local_ranks;
    const int op = op_code(op_obj);
    if (op < 0) return nullptr;
    if (outs.single != inps.single || outs.size != n || inps.size != n) {
        PyErr_Format(PyExc_ValueError, "need one tensor per local rank (%d)", n);
        return nullptr;
    }
    const char* what[] = {"input", "output"};
    PyObject* firsts[] = {inps.item[0], outs.item[0]};
    for (int k = 0; k < 2; ++k) {
        if (!THPVariable_Check(firsts[k])) {
            PyErr_Format(PyExc_ValueError, "%s[0] must be a contiguous CUDA tensor", what[k]);
            return nullptr;
        }
    }
    const at::Tensor& first_in = THPVariable_Unpack(firsts[0]);
    const at::Tensor& first_out = THPVariable_Unpack(firsts[1]);
    const at::ScalarType dtype = first_in.scalar_type();
    const std::int64_t in_numel = first_in.numel();
    std::int64_t out_numel = in_numel, count = in_numel;
    if (collective == 1) {
        out_numel = count = first_out.numel();
        if (in_numel != out_numel * c->world) {
            PyErr_SetString(PyExc_ValueError, "reduce_scatter: input must hold world_size blocks of the output's size");
            return nullptr;
        }
    } else if (collective == 2) {
        out_numel = first_out.numel();
        if (out_numel != in_numel * c->world) {
            PyErr_SetString(PyExc_ValueError, "all_gather: output must hold world_size blocks of the input's size");
            return nullptr;
        }
    }
    const int code = dtype_code(dtype);
    if (code < 0) {
        PyObject* d = PyObject_GetAttrString(firsts[0], "dtype");
        if (d != nullptr) PyErr_Format(PyExc_ValueError, "unsupported dtype %S", d);
        Py_XDECREF(d);
        return nullptr;
    }
    void *send[kMaxRanks], *recv[kMaxRanks], *streams[kMaxRanks];
    for (int i = 0; i < n; ++i) {
        if (!check_tensor("input", i, inps.item[i], dtype, in_numel, c->device[i]) ||
            !check_tensor("output", i, outs.item[i], dtype, out_numel, c->device[i]))
            return nullptr;
        send[i] = THPVariable_Unpack(inps.item[i]).data_ptr();
        recv[i] = THPVariable_Unpack(outs.item[i]).data_ptr();
    }
    if (!read_streams(c, streams_obj, inps.single, streams)) return nullptr;
    const int in_place = collective == 0 && send[0] == recv[0] ? 1 : 0;
    int rc;
    // Other Python threads run meanwhile: the launch may block on a full queue, and ranks of one job
    // that live in several threads of one process meet inside their first calls.
    Py_BEGIN_ALLOW_THREADS
    rc = g_collective(c->handle, collective, send, recv, streams, static_cast<std::size_t>(count), code, op, in_place);
    Py_END_ALLOW_THREADS
    if (rc != 0) {
        PyErr_SetString(rc == 2 ? PyExc_ValueError : g_error_class, g_last_error());
        return nullptr;
    }
    Py_INCREF(outs_obj);
    return outs_obj;
}

PyObject* guarded_run(PyObject* self, int collective, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 4) {
        PyErr_SetString(PyExc_TypeError, "expected (out, inp, op, stream)");
        return nullptr;
    }
    try {
        return run(reinterpret_cast<Caller*>(self), collective, args[0], args[1], args[2], args[3]);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyObject* caller_all_reduce(PyObject* s, PyObject* const* a, Py_ssize_t n) { return guarded_run(s, 0, a, n); }
PyObject* caller_reduce_scatter(PyObject* s, PyObject* const* a, Py_ssize_t n) { return guarded_run(s, 1, a, n); }
PyObject* caller_all_gather(PyObject* s, PyObject* const* a, Py_ssize_t n) { return guarded_run(s, 2, a, n); }
PyObject* caller_close(PyObject* s, PyObject*) {
    reinterpret_cast<Caller*>(s)->handle = nullptr;
    Py_RETURN_NONE;
}

PyMethodDef caller_methods[] = {
    {"all_reduce", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(caller_all_reduce)), METH_FASTCALL, nullptr},
    {"reduce_scatter", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(caller_reduce_scatter)), METH_FASTCALL, nullptr},
    {"all_gather", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(caller_all_gather)), METH_FASTCALL, nullptr},
    {"close", caller_close, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};

// Caller(handle, devices, world_size): `devices` holds the GPU of every local rank.
PyObject* caller_new(PyTypeObject* type, PyObject* args, PyObject*) {
    unsigned long long handle = 0;
    PyObject* devices = nullptr;
    long long world = 0;
    if (!PyArg_ParseTuple(args, "KO!L", &handle, &PyTuple_Type, &devices, &world)) return nullptr;
    const Py_ssize_t n = PyTuple_GET_SIZE(devices);
    if (g_collective == nullptr || handle == 0 || n < 1 || n > kMaxRanks) {
        PyErr_SetString(PyExc_ValueError, "Caller: bind() first, then a live communicator with one device per local rank");
        return nullptr;
    }
    Caller* c = reinterpret_cast<Caller*>(type->tp_alloc(type, 0));
    if (c == nullptr) return nullptr;
    c->handle = reinterpret_cast<void*>(static_cast<std::uintptr_t>(handle));
    c->local_ranks = static_cast<int>(n);
    c->world = world;
    for (Py_ssize_t i = 0; i < n; ++i) {
        c->device[i] = static_cast<int>(PyLong_AsLong(PyTuple_GET_ITEM(devices, i)));
        if (PyErr_Occurred()) {
            Py_DECREF(c);
            return nullptr;
        }
    }
    return reinterpret_cast<PyObject*>(c);
}

PyType_Slot caller_slots[] = {{Py_tp_methods, caller_methods}, {Py_tp_new, reinterpret_cast<void*>(caller_new)}, {0, nullptr}};
PyType_Spec caller_spec = {"_b200ccl_torch.Caller", sizeof(Caller), 0, Py_TPFLAGS_DEFAULT, caller_slots};

// bind(address of b2_collective, address of b2_last_error, exception class)
PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long collective = 0, last_error = 0;
    PyObject* cls = nullptr;
    if (!PyArg_ParseTuple(args, "KKO", &collective, &last_error, &cls)) return nullptr;
    g_collective = reinterpret_cast<CollectiveFn>(static_cast<std::uintptr_t>(collective));
    g_last_error = reinterpret_cast<LastErrorFn>(static_cast<std::uintptr_t>(last_error));
    Py_INCREF(cls);
    Py_XSETREF(g_error_class, cls);
    Py_RETURN_NONE;
}

PyMethodDef module_methods[] = {{"bind", bind, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_b200ccl_torch", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200ccl_torch() {
    PyObject* m = PyModule_Create(&module_def);
    if (m == nullptr) return nullptr;
    PyObject* type = PyType_FromSpec(&caller_spec);
    if (type == nullptr || PyModule_AddObject(m, "Caller", type) < 0) {
        Py_XDECREF(type);
        Py_DECREF(m);
        return nullptr;
    }
    // The calls read torch's own structures: whoever loads the module compares this with the torch that runs.
    if (PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
