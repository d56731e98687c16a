// Native front end of gdn_chunk: the argument checks, output allocation and the call of the C ABI that the Python wrapper
// (gdn_chunk_interface.py) would make, without its interpreter time (about 20 of the 27 microseconds of a one-token call).
//
// Only the plain case is handled here: CUDA tensors of the current device, contiguous, in the dtypes the kernels read.
// Anything else - conversions, other devices, wrong shapes and their error messages - returns None and takes the Python
// wrapper, so both behave the same.  The module is a CPython extension that links the kernel library.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>

#include "../../include/gdn_chunk_sm100.h"

namespace {

// Scratch buffers by (device, stream), handed over by the Python wrapper, which owns the policy (one per device and stream,
// grown when too small).  Guarded by the interpreter lock; a call keeps its own reference, since the lock is released while
// it enqueues and another thread may put a larger buffer in place meanwhile.
std::map<std::pair<int, void*>, at::Tensor>& scratch_buffers() {
    static auto* m = new std::map<std::pair<int, void*>, at::Tensor>;   // lives as long as the process: no CUDA calls at exit
    return *m;
}
PyObject* g_grow_scratch = nullptr;   // _scratch_for(device index, bytes), which calls note_scratch

// Releases the interpreter lock: a launch may block on a full queue behind work that needs it, an allocation may synchronise.
class Unlocked {
public:
    Unlocked() : state_(PyEval_SaveThread()) {}
    ~Unlocked() { PyEval_RestoreThread(state_); }
    Unlocked(const Unlocked&) = delete;
    Unlocked& operator=(const Unlocked&) = delete;

private:
    PyThreadState* state_;
};

bool plain(const at::Tensor& t, at::ScalarType dtype, const at::Device& dev) {
    return t.defined() && t.scalar_type() == dtype && t.device() == dev && t.layout() == at::kStrided && t.is_contiguous() && !t.is_neg() &&
           !t.is_conj();
}

PyObject* forward_plain(PyObject* const* a, Py_ssize_t n) {
    if (n != 10) {
        PyErr_SetString(PyExc_TypeError, "forward takes 10 arguments");
        return nullptr;
    }
    for (int i = 0; i < 5; ++i)
        if (!THPVariable_Check(a[i])) Py_RETURN_NONE;
    const at::Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]),
                     &g = THPVariable_Unpack(a[3]), &beta = THPVariable_Unpack(a[4]);
    if (!q.defined() || !q.is_cuda() || q.dim() != 4 || v.dim() != 4 || g.dim() != 3) Py_RETURN_NONE;
    const at::Device dev = q.device();
    if (c10::cuda::current_device() != dev.index()) Py_RETURN_NONE;
    if (!plain(q, at::kBFloat16, dev) || !plain(k, at::kBFloat16, dev) || !plain(v, at::kBFloat16, dev)) Py_RETURN_NONE;
    const at::ScalarType gate = g.scalar_type();
    if ((gate != at::kBFloat16 && gate != at::kFloat) || !plain(g, gate, dev) || !plain(beta, gate, dev)) Py_RETURN_NONE;
    const int64_t B = q.size(0), S = q.size(1), Hk = q.size(2), Hv = v.size(2);
    if (B <= 0 || S <= 0 || Hk <= 0 || Hv <= 0 || B > INT32_MAX || S > INT32_MAX || Hv > INT32_MAX) Py_RETURN_NONE;
    if (q.size(3) != GDN_D || k.sizes() != q.sizes() || v.size(0) != B || v.size(1) != S || v.size(3) != GDN_D || Hv % Hk != 0) Py_RETURN_NONE;
    if (g.size(0) != B || g.size(1) != S || g.size(2) != Hv || beta.sizes() != g.sizes()) Py_RETURN_NONE;

    const int want_state = PyObject_IsTrue(a[5]);
    if (want_state < 0) return nullptr;
    const float* h0 = nullptr;
    if (a[6] != Py_None) {
        if (!THPVariable_Check(a[6])) Py_RETURN_NONE;
        const at::Tensor& t = THPVariable_Unpack(a[6]);
        if (!plain(t, at::kFloat, dev) || t.dim() != 4 || t.size(0) != B || t.size(1) != Hv || t.size(2) != GDN_D || t.size(3) != GDN_D) Py_RETURN_NONE;
        h0 = t.const_data_ptr<float>();
    }
    const long path = PyLong_AsLong(a[7]), flags = PyLong_AsLong(a[8]);
    if (PyErr_Occurred()) return nullptr;

    const void *z = nullptr, *w = nullptr;
    double eps = 1e-6;
    if (a[9] != Py_None) {
        if (!PyTuple_CheckExact(a[9])) Py_RETURN_NONE;
        const Py_ssize_t m = PyTuple_GET_SIZE(a[9]);
        if (m != 2 && m != 3) Py_RETURN_NONE;
        PyObject *pz = PyTuple_GET_ITEM(a[9], 0), *pw = PyTuple_GET_ITEM(a[9], 1);
        if (!THPVariable_Check(pz) || !THPVariable_Check(pw)) Py_RETURN_NONE;
        const at::Tensor &tz = THPVariable_Unpack(pz), &tw = THPVariable_Unpack(pw);
        if (!plain(tz, at::kBFloat16, dev) || !plain(tw, at::kBFloat16, dev) || tz.sizes() != v.sizes() || tw.numel() != GDN_D) Py_RETURN_NONE;
        if (m == 3) {
            eps = PyFloat_AsDouble(PyTuple_GET_ITEM(a[9], 2));
            if (PyErr_Occurred()) return nullptr;
        }
        z = tz.const_data_ptr();
        w = tw.const_data_ptr();
    }
    const char* check = std::getenv("GDN_CHUNK_CHECK_STATUS");
    if (check && !std::strcmp(check, "1")) Py_RETURN_NONE;

    void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const size_t need = gdn_chunk_scratch_bytes(static_cast<int>(B), static_cast<int>(S), static_cast<int>(Hk), static_cast<int>(Hv), static_cast<int>(path));
    auto& buffers = scratch_buffers();
    auto it = buffers.find({dev.index(), stream});
    if (it == buffers.end() || static_cast<size_t>(it->second.numel()) < need) {
        if (!g_grow_scratch) Py_RETURN_NONE;
        PyObject* r = PyObject_CallFunction(g_grow_scratch, "in", static_cast<int>(dev.index()), static_cast<Py_ssize_t>(need));
        if (!r) return nullptr;
        Py_DECREF(r);
        it = buffers.find({dev.index(), stream});
        if (it == buffers.end() || static_cast<size_t>(it->second.numel()) < need) Py_RETURN_NONE;
    }
    const at::Tensor buffer = it->second;
    void* scratch = buffer.data_ptr();
    const size_t scratch_bytes = static_cast<size_t>(buffer.numel());

    const void *qp = q.const_data_ptr(), *kp = k.const_data_ptr(), *vp = v.const_data_ptr(), *gp = g.const_data_ptr(), *bp = beta.const_data_ptr();
    const int gate_code = gate == at::kFloat ? GDN_GATE_F32 : GDN_GATE_BF16;
    at::Tensor out, hT;
    int st;
    {
        const Unlocked unlocked;   // (its destructor runs before an exception reaches the handler)
        out = at::Tensor(at::detail::empty_cuda({B, S, Hv, GDN_D}, at::kBFloat16, dev, std::nullopt));
        if (want_state) hT = at::Tensor(at::detail::empty_cuda({B, Hv, GDN_D, GDN_D}, at::kFloat, dev, std::nullopt));
        float* state = want_state ? hT.mutable_data_ptr<float>() : nullptr;
        st = z ? gdn_chunk_fwd_gated_sm100(qp, kp, vp, gp, bp, h0, z, w, static_cast<float>(eps), out.mutable_data_ptr(), state, scratch,
                                           scratch_bytes, static_cast<int>(B), static_cast<int>(S), static_cast<int>(Hk), static_cast<int>(Hv),
                                           gate_code, static_cast<int>(path), static_cast<unsigned>(flags), stream)
               : gdn_chunk_fwd_sm100_ex(qp, kp, vp, gp, bp, h0, out.mutable_data_ptr(), state, scratch, scratch_bytes, static_cast<int>(B),
                                        static_cast<int>(S), static_cast<int>(Hk), static_cast<int>(Hv), gate_code, static_cast<int>(path),
                                        static_cast<unsigned>(flags), stream);
    }
    if (st != GDN_OK) Py_RETURN_NONE;   // the wrapper makes the call again and raises its status
    PyObject* po = THPVariable_Wrap(std::move(out));
    if (!po) return nullptr;
    PyObject* ps = Py_None;
    if (want_state) ps = THPVariable_Wrap(std::move(hT));
    else Py_INCREF(ps);
    if (!ps) {
        Py_DECREF(po);
        return nullptr;
    }
    PyObject* r = PyTuple_New(2);
    if (!r) {
        Py_DECREF(po);
        Py_DECREF(ps);
        return nullptr;
    }
    PyTuple_SET_ITEM(r, 0, po);
    PyTuple_SET_ITEM(r, 1, ps);
    return r;
}

// forward(q, k, v, g, beta, output_final_state, initial_state, path, flags, output_gate) -> (out, state) or None
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    // tensors without storage (fake, batched, nested) throw when their size or address is asked for; no exception may
    // leave a function the interpreter called, and the wrapper meets the same error and reports it
    try {
        return forward_plain(a, n);
    } catch (...) {
        if (PyErr_Occurred()) return nullptr;
        Py_RETURN_NONE;
    }
}

// note_scratch(device index, stream handle, tensor): the buffer calls on that stream use from now on
PyObject* note_scratch(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 3 || !THPVariable_Check(a[2])) {
        PyErr_SetString(PyExc_TypeError, "note_scratch(device index, stream handle, tensor)");
        return nullptr;
    }
    const long dev = PyLong_AsLong(a[0]);
    void* stream = PyLong_AsVoidPtr(a[1]);
    if (PyErr_Occurred()) return nullptr;
    scratch_buffers()[{static_cast<int>(dev), stream}] = THPVariable_Unpack(a[2]);
    Py_RETURN_NONE;
}

PyObject* set_grow_scratch(PyObject*, PyObject* fn) {
    Py_INCREF(fn);
    Py_XDECREF(g_grow_scratch);
    g_grow_scratch = fn;
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(forward)), METH_FASTCALL, "the forward pass, or None when the call is not a plain one"},
    {"note_scratch", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(note_scratch)), METH_FASTCALL, "hands over a scratch buffer"},
    {"set_grow_scratch", set_grow_scratch, METH_O, "the function that grows a scratch buffer"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_gdn_frontend", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__gdn_frontend(void) {
    PyObject* m = PyModule_Create(&module_def);
    if (m && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) {   // what it was built against
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
