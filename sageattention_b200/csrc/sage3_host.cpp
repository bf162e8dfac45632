// Host side of the functional entry points as a CPython extension: argument checks, output and workspace tensors, and the one
// call into the C ABI.  The same steps in Python (signature lookup, two allocations, stream and device queries, ctypes
// conversion) took 19 us of the 32 us a call needs on the host, and a call of 1 024 tokens takes less than that on the GPU.
// Anything unusual (copies needed, per-head scale, wrong types or shapes) returns None: the Python path deals with it and raises
// what there is to raise.
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <ATen/ops/full.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <limits>
#include <map>
#include <mutex>
#include <utility>

#include "../../include/sage3_b200.h"

namespace {

using FwdFn = int (*)(const Sage3Desc*, const void*, const void*, const void*, void*, void*, float*, void*);
using VarlenFn = int (*)(const Sage3Desc*, const int32_t*, const int32_t*, const void*, const void*, const void*, void*, float*, void*, void*);
using BytesFn = size_t (*)(const Sage3Desc*);
FwdFn g_fwd = nullptr;
VarlenFn g_varlen = nullptr;
BytesFn g_bytes = nullptr;

// One workspace per (device, stream), grown on demand and reused by later calls: kernels of successive calls on one stream
// run in order, so they may share it (sage3_fwd and sage3_fwd_varlen enqueue a call as a whole, also when several threads use the
// stream; a buffer that was replaced meanwhile lives as long as the call that holds it); calls on different streams get different
// buffers.  (Allocating 3.4 GB anew on every call of the 4 x 32 x 32 768 shape costs more than the pre-pass.)
std::mutex g_mutex;
std::map<std::pair<int, cudaStream_t>, at::Tensor>* g_workspaces = nullptr;      // never destroyed: the CUDA context may go first

at::Tensor workspace(int device, cudaStream_t stream, size_t bytes) {      // (the device and its stream are the current ones)
    const auto options = at::TensorOptions().dtype(at::kByte).device(at::Device(at::kCUDA, device));
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return at::empty({(int64_t)bytes}, options);
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_workspaces) g_workspaces = new std::map<std::pair<int, cudaStream_t>, at::Tensor>();
    at::Tensor& t = (*g_workspaces)[{device, stream}];
    if (!t.defined() || (size_t)t.numel() < bytes) {
        t = at::Tensor();                             // give the old one back first
        t = at::empty({(int64_t)bytes}, options);
    }
    return t;
}

void* aligned_base(const at::Tensor& t) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(t.data_ptr());
    return reinterpret_cast<void*>((p + 255) & ~uintptr_t(255));
}

// rows the kernels can load as they are: contiguous last dimension, 16-byte aligned rows
bool usable(const at::Tensor& t) {
    const auto st = t.strides();
    const size_t n = st.size();
    if (st[n - 1] != 1) return false;
    for (size_t i = 0; i + 1 < n; ++i)
        if (st[i] % 8 != 0 || st[i] < 0) return false;
    return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

bool same_kind(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
    if (!q.is_cuda() || !k.is_cuda() || !v.is_cuda()) return false;
    const auto dt = q.scalar_type();
    if ((dt != at::kHalf && dt != at::kBFloat16) || k.scalar_type() != dt || v.scalar_type() != dt) return false;
    return k.device() == q.device() && v.device() == q.device();
}

// 0 asks for the default; any other scale has to be positive as the 32-bit value of the descriptor, too (1e-60 is not)
bool scale_ok(double scale) { return scale == 0 || (float)scale > 0; }

PyObject* result(const at::Tensor& out, const at::Tensor& lse) {
    if (!lse.defined()) return THPVariable_Wrap(out);
    PyObject* t = PyTuple_New(2);
    if (!t) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(out));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(lse));
    return t;
}

bool truth(PyObject* o, bool* out) {
    const int v = PyObject_IsTrue(o);
    *out = v == 1;
    return v >= 0;
}

// fwd(q, k, v, nhd, is_causal, scale (0: default), per_block_mean, return_lse) -> out | (out, lse) | status code | None
PyObject* fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8 || !g_fwd) Py_RETURN_NONE;
    for (int i = 0; i < 3; ++i)
        if (!THPVariable_CheckExact(args[i])) Py_RETURN_NONE;
    const at::Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
    bool nhd, causal, block_mean, want_lse;
    if (!truth(args[3], &nhd) || !truth(args[4], &causal) || !truth(args[6], &block_mean) || !truth(args[7], &want_lse)) return nullptr;
    const double scale = PyFloat_AsDouble(args[5]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
    if (!scale_ok(scale) || q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || !same_kind(q, k, v)) Py_RETURN_NONE;
    const int hd = nhd ? 2 : 1, nd = nhd ? 1 : 2;
    const auto qs = q.sizes(), ks = k.sizes();
    const int64_t B = qs[0], Hq = qs[hd], Nq = qs[nd], D = qs[3], Hkv = ks[hd], Nk = ks[nd];
    const int64_t most = std::numeric_limits<int32_t>::max();
    if (ks[0] != B || v.sizes() != ks || ks[3] != D || (D != 64 && D != 128) || Hkv <= 0 || Hq <= 0 || Hq % Hkv != 0 || B <= 0 || Nq <= 0 ||
        Nk <= 0 || B > most || Hq > most || Nq > most || Nk > most || !usable(q) || !usable(k) || !usable(v))
        Py_RETURN_NONE;
    Sage3Desc d = {};
    d.B = (int32_t)B; d.Hq = (int32_t)Hq; d.Hkv = (int32_t)Hkv; d.Nq = (int32_t)Nq; d.Nk = (int32_t)Nk; d.D = (int32_t)D;
    d.dtype = q.scalar_type() == at::kBFloat16 ? SAGE3_BF16 : SAGE3_FP16;
    d.is_causal = causal;
    d.per_block_mean = block_mean;
    d.sm_scale = (float)scale;
    const c10::cuda::CUDAGuard guard(q.device());
    const at::Tensor out = at::empty(qs, q.options());
    const at::Tensor lse = want_lse ? at::empty({B, Hq, Nq}, q.options().dtype(at::kFloat)) : at::Tensor();
    auto strides = [&](const at::Tensor& t, int64_t* s) {
        const auto st = t.strides();
        s[0] = st[0]; s[1] = st[hd]; s[2] = st[nd];
    };
    strides(q, d.q_stride); strides(k, d.k_stride); strides(v, d.v_stride); strides(out, d.o_stride);
    const size_t bytes = g_bytes(&d);
    if (bytes == 0) Py_RETURN_NONE;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    const at::Tensor ws = workspace(q.device().index(), stream, bytes + 256);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_fwd(&d, q.data_ptr(), k.data_ptr(), v.data_ptr(), aligned_base(ws), out.data_ptr(), want_lse ? lse.data_ptr<float>() : nullptr, stream);
    Py_END_ALLOW_THREADS
    return rc == SAGE3_OK ? result(out, lse) : PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// fwd_varlen(q, k, v, cu_q, cu_k, max_q, max_k, is_causal, scale (0: default), per_block_mean, return_lse), likewise
PyObject* fwd_varlen(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 11 || !g_varlen) Py_RETURN_NONE;
    for (int i = 0; i < 5; ++i)
        if (!THPVariable_CheckExact(args[i])) Py_RETURN_NONE;
    const at::Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
    const at::Tensor &cq = THPVariable_Unpack(args[3]), &ck = THPVariable_Unpack(args[4]);
    const long max_q = PyLong_AsLong(args[5]), max_k = PyLong_AsLong(args[6]);
    const double scale = PyFloat_AsDouble(args[8]);
    if (PyErr_Occurred()) return nullptr;
    bool causal, block_mean, want_lse;
    if (!truth(args[7], &causal) || !truth(args[9], &block_mean) || !truth(args[10], &want_lse)) return nullptr;
    if (!scale_ok(scale) || q.dim() != 3 || k.dim() != 3 || v.dim() != 3 || !same_kind(q, k, v)) Py_RETURN_NONE;
    for (const at::Tensor* c : {&cq, &ck})
        if (!c->is_cuda() || c->device() != q.device() || c->scalar_type() != at::kInt || c->dim() != 1 || !c->is_contiguous()) Py_RETURN_NONE;
    const int64_t Hq = q.size(1), Hkv = k.size(1), D = q.size(2), nseq = cq.size(0) - 1;
    const int64_t most = std::numeric_limits<int32_t>::max();
    if (v.sizes() != k.sizes() || k.size(2) != D || (D != 64 && D != 128) || Hkv <= 0 || Hq <= 0 || Hq % Hkv != 0 || nseq < 1 || ck.size(0) != nseq + 1 ||
        q.size(0) == 0 || k.size(0) == 0 || max_q < 1 || max_k < 1 || max_q > most || max_k > most || !usable(q) || !usable(k) || !usable(v))
        Py_RETURN_NONE;
    Sage3Desc d = {};
    d.reserved = SAGE3_NO_SHARED_TILES;                // (a packed batch shares none)
    d.B = (int32_t)nseq; d.Hq = (int32_t)Hq; d.Hkv = (int32_t)Hkv; d.Nq = (int32_t)max_q; d.Nk = (int32_t)max_k; d.D = (int32_t)D;
    d.dtype = q.scalar_type() == at::kBFloat16 ? SAGE3_BF16 : SAGE3_FP16;
    d.is_causal = causal;
    d.per_block_mean = block_mean;
    d.sm_scale = (float)scale;
    const c10::cuda::CUDAGuard guard(q.device());
    const at::Tensor out = at::empty_like(q);          // (the strides of a permuted q, as on the Python path)
    const at::Tensor lse = want_lse ? at::full({nseq, Hq, (int64_t)max_q}, -std::numeric_limits<double>::infinity(), q.options().dtype(at::kFloat))
                                    : at::Tensor();
    auto strides = [&](const at::Tensor& t, int64_t* s) {
        s[0] = 0; s[1] = t.stride(1); s[2] = t.stride(0);
    };
    strides(q, d.q_stride); strides(k, d.k_stride); strides(v, d.v_stride); strides(out, d.o_stride);
    const size_t bytes = g_bytes(&d);
    if (bytes == 0) Py_RETURN_NONE;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    const at::Tensor ws = workspace(q.device().index(), stream, bytes + 256);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_varlen(&d, cq.data_ptr<int32_t>(), ck.data_ptr<int32_t>(), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                  want_lse ? lse.data_ptr<float>() : nullptr, aligned_base(ws), stream);
    Py_END_ALLOW_THREADS
    return rc == SAGE3_OK ? result(out, lse) : PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// shared_buffer(device index, bytes) -> the current stream's workspace
PyObject* shared_buffer(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2) {
        PyErr_SetString(PyExc_TypeError, "shared_buffer(device index, bytes)");
        return nullptr;
    }
    const long dev = PyLong_AsLong(args[0]);
    const long long bytes = PyLong_AsLongLong(args[1]);
    if (PyErr_Occurred()) return nullptr;
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    return THPVariable_Wrap(workspace((int)dev, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(), (size_t)bytes));
    END_HANDLE_TH_ERRORS
}

PyObject* release(PyObject*, PyObject*) {
    HANDLE_TH_ERRORS
    std::map<std::pair<int, cudaStream_t>, at::Tensor> gone;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        if (g_workspaces) gone.swap(*g_workspaces);
    }
    gone.clear();
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// bind(address of sage3_fwd, of sage3_fwd_varlen, of sage3_workspace_bytes)
PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long a, b, c;
    if (!PyArg_ParseTuple(args, "KKK", &a, &b, &c)) return nullptr;
    g_fwd = reinterpret_cast<FwdFn>(a);
    g_varlen = reinterpret_cast<VarlenFn>(b);
    g_bytes = reinterpret_cast<BytesFn>(c);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"fwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fwd)), METH_FASTCALL, nullptr},
    {"fwd_varlen", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fwd_varlen)), METH_FASTCALL, nullptr},
    {"shared_buffer", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(shared_buffer)), METH_FASTCALL, nullptr},
    {"release", release, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host(void) { return PyModule_Create(&module); }
