// Host side of one QuantLinear.forward call in native code.
//
// A decode GEMV runs for 3..10 us on the device; preparing its launch from Python (attribute look-ups, argument
// conversion of a ctypes call, torch.empty) took 12..16 us per call and the GEMM's 27..31 us, so a loop of small calls
// was bound by the host.  This module does the same checks and the same library call from C++: `Layer.run(x,
// module.__dict__)` returns the output tensor, or None when anything about the call is not the prepared case (another
// device, other buffers, a row count without a plan, a tensor subclass); the caller then takes the Python route,
// which prepares what is missing.  Nothing here launches kernels of its own: the work goes through the C ABI.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <unordered_map>

#include "../../../../include/b200gptq.h"

namespace {

constexpr int kMaxGemvRows = 16;

// Scratch buffers by (device, stream), registered by ops.get_workspace.  Read and written under the GIL; `owner` is the
// tensor, held while it is registered and by a call that works without the GIL.  in_graph: it was handed out while its stream
// was being captured, so a graph may hold its address for good.
struct Scratch { PyObject* owner; void* ptr; size_t bytes; bool in_graph; };
struct KeyHash {
    size_t operator()(const std::pair<int, void*>& k) const {
        return std::hash<void*>()(k.second) * 31u + (size_t)k.first;
    }
};
std::unordered_map<std::pair<int, void*>, Scratch, KeyHash>* g_scratch;
PyObject* g_get_workspace;   // ops.get_workspace, for a stream without a large enough buffer

PyObject *s_buffers, *s_qweight, *s_g_idx, *s_qzeros, *s_scales, *s_bias, *s_gemv_tuning;

struct GemvEntry {
    PyObject* owner;      // the ops.GemvPlan that owns the handle
    const b200gptq_gemv_plan* plan;
    size_t need;
};

struct Layer {
    PyObject_HEAD
    int K, N, bits, group_size, device;
    // the buffers this object was prepared for: addresses of qweight / g_idx, identity and addresses of the others, and how
    // often the weights, scales and zero-points had been written to
    const void *qweight_at, *g_idx_at;
    uint32_t writes;
    PyObject *qzeros, *scales, *bias, *tuning;
    GemvEntry gemv[kMaxGemvRows + 1];
    // run-time layout for the GEMM (gemm_ok false: no tensor-core kernel for this layer)
    bool gemm_ok;
    int gemv_rows;        // largest row count that goes through plans (8, or 16 where the streaming kernel takes the layer)
    const int32_t *qweight_run, *qzeros_run, *g_idx_run, *x_perm;
    const void *scales_run, *bias_run;
    PyObject* keep;       // keeps the tensors behind those addresses alive
};

// A reference held for the time of a call.
struct Held {
    PyObject* o;
    explicit Held(PyObject* p) : o(p) { Py_XINCREF(o); }
    ~Held() { Py_XDECREF(o); }
    Held(const Held&) = delete;
    Held& operator=(const Held&) = delete;
};
// The GIL given up for the time of a scope.
struct WithoutGil {
    PyThreadState* state = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

// Tensors that stand for something else: wrappers without memory of their own (vmap, grad and their kin), views whose values
// are not what lies in memory.
const c10::DispatchKeySet kNotPlain({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::BatchedNestedTensor,
                                     c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                     c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});

inline const void* tensor_address(PyObject* t) {
    return t && t != Py_None && THPVariable_Check(t) ? THPVariable_Unpack(t).unsafeGetTensorImpl()->data() : nullptr;
}
// Writes in place to a tensor so far (tensors of inference mode do not count them).
inline uint32_t writes_to(PyObject* t) {
    c10::TensorImpl* impl = THPVariable_Unpack(t).unsafeGetTensorImpl();
    return impl->is_inference() ? 0u : impl->version_counter().current_version();
}
inline bool lies_at(PyObject* t, const void* at) {
    return t && THPVariable_Check(t) && THPVariable_Unpack(t).unsafeGetTensorImpl()->data() == at;
}

// (the legacy default stream cannot be captured)
bool is_capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (stream) C10_CUDA_CHECK(cudaStreamIsCapturing(stream, &status));
    return status != cudaStreamCaptureStatusNone;
}

bool scratch_for(int device, cudaStream_t stream, size_t need, Scratch* out) {
    auto it = g_scratch->find({device, (void*)stream});
    if (it != g_scratch->end() && !it->second.in_graph) it->second.in_graph = is_capturing(stream);
    if (it == g_scratch->end() || it->second.bytes < need) {
        PyObject* r = PyObject_CallFunction(g_get_workspace, "in", device, (Py_ssize_t)need);
        if (!r) return false;
        Py_DECREF(r);
        it = g_scratch->find({device, (void*)stream});
        if (it == g_scratch->end() || it->second.bytes < need) {
            PyErr_SetString(PyExc_RuntimeError, "no scratch buffer was registered for this stream");
            return false;
        }
    }
    *out = it->second;
    return true;
}

// The module's forward, or None where the prepared case does not apply.
PyObject* run_prepared(Layer* self, PyObject* px, PyObject* dict) {
    if (!THPVariable_CheckExact(px) || !PyDict_Check(dict)) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(px);
    if (x.key_set().has_any(kNotPlain)) Py_RETURN_NONE;
    const int64_t dims = x.dim();
    if (!x.is_cuda() || x.scalar_type() != at::kHalf || dims < 1 || x.size(-1) != self->K || !x.is_contiguous() ||
        x.get_device() != self->device)
        Py_RETURN_NONE;
    const int64_t M = x.numel() / self->K;
    if (M < 1) Py_RETURN_NONE;
    // the module's buffers are the ones this object was prepared for
    PyObject* buffers = PyDict_GetItem(dict, s_buffers);
    if (!buffers) Py_RETURN_NONE;
    PyObject *qweight = PyDict_GetItem(buffers, s_qweight), *g_idx = PyDict_GetItem(buffers, s_g_idx);
    if (!lies_at(qweight, self->qweight_at) || !lies_at(g_idx, self->g_idx_at)) Py_RETURN_NONE;
    PyObject* bias = PyDict_GetItem(buffers, s_bias);
    if (!bias) bias = PyDict_GetItem(dict, s_bias);
    if ((bias ? bias : Py_None) != self->bias || PyDict_GetItem(buffers, s_qzeros) != self->qzeros ||
        PyDict_GetItem(buffers, s_scales) != self->scales)
        Py_RETURN_NONE;
    // (`tensor.data = other` keeps the tensor and moves its numbers)
    auto at = [](PyObject* t) { return THPVariable_Unpack(t).unsafeGetTensorImpl()->data(); };
    if (at(self->qzeros) != self->qzeros_run || at(self->scales) != self->scales_run ||
        (self->bias_run && at(self->bias) != self->bias_run))
        Py_RETURN_NONE;
    // (weights that have been written to: the Python route re-orders them anew, or sees to it that they can be read early)
    if (writes_to(qweight) + writes_to(g_idx) + writes_to(self->qzeros) + writes_to(self->scales) != self->writes) Py_RETURN_NONE;
    const bool gemv = M <= self->gemv_rows;
    const GemvEntry* e = gemv ? &self->gemv[M] : nullptr;
    if (gemv ? (!e->plan || PyDict_GetItem(dict, s_gemv_tuning) != self->tuning) : !self->gemm_ok) Py_RETURN_NONE;
    if (c10::cuda::current_device() != self->device || M > INT32_MAX) Py_RETURN_NONE;

    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream();
    Scratch ws;
    const size_t need = gemv ? e->need : b200gptq_workspace_bytes(B200GPTQ_OP_GEMM, (int)M, self->K, self->N, self->bits);
    if (!scratch_for(self->device, stream, need, &ws)) return nullptr;
    // What another thread may replace while this one has given up the GIL.  (`self`, its tensors and x are held by the caller.)
    const b200gptq_gemv_plan* plan = gemv ? e->plan : nullptr;
    const Held scratch(ws.owner), owner(gemv ? e->owner : nullptr);
    c10::SmallVector<int64_t, 4> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = self->N;
    at::Tensor y;
    int st;
    {
        // A launch waits while the device's queue is full, an allocation may wait for the device: other threads go on.
        const WithoutGil released;
        y = at::detail::empty_cuda(shape, at::kHalf, at::Device(at::kCUDA, (c10::DeviceIndex)self->device), std::nullopt);
        const void* xp = x.unsafeGetTensorImpl()->data();
        void* yp = y.unsafeGetTensorImpl()->mutable_data();
        if (gemv)
            st = b200gptq_gemv_plan_run(plan, xp, yp, ws.ptr, ws.bytes, stream);
        else
            st = b200gptq_gemm(xp, self->qweight_run, self->qzeros_run, self->scales_run, self->g_idx_run, self->x_perm,
                               self->bias_run, yp, (int)M, self->K, self->N, self->bits, self->group_size, ws.ptr, ws.bytes,
                               stream);
    }
    if (st != B200GPTQ_OK) Py_RETURN_NONE;   // the Python route repeats the call and reports the status
    return THPVariable_Wrap(std::move(y));
}

// Layer.run(x, module_dict).  No C++ exception leaves here: out of memory, or a tensor that has no address, is met again by
// the Python route, which raises it with its own type.
PyObject* layer_run(PyObject* self_, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "run(x, module_dict)"); return nullptr; }
    try {
        return run_prepared(reinterpret_cast<Layer*>(self_), args[0], args[1]);
    } catch (const std::exception&) {
        Py_RETURN_NONE;
    }
}

// Layer.set_gemv(rows, plan_owner, plan_handle, workspace_bytes)
PyObject* layer_set_gemv(PyObject* self_, PyObject* args) {
    Layer* self = reinterpret_cast<Layer*>(self_);
    int rows;
    PyObject* owner;
    unsigned long long handle, need;
    if (!PyArg_ParseTuple(args, "iOKK", &rows, &owner, &handle, &need)) return nullptr;
    if (rows < 1 || rows > kMaxGemvRows) { PyErr_SetString(PyExc_ValueError, "rows"); return nullptr; }
    GemvEntry& e = self->gemv[rows];
    Py_INCREF(owner);
    Py_XSETREF(e.owner, owner);
    e.plan = reinterpret_cast<const b200gptq_gemv_plan*>((uintptr_t)handle);
    e.need = (size_t)need;
    Py_RETURN_NONE;
}

// Layer(K, N, bits, group_size, device, module_dict, gemm_ok, gemv_rows, qweight_run, g_idx_run, x_perm)
PyObject* make_layer(PyTypeObject* type, PyObject* args) {
    int K, N, bits, group_size, device, gemm_ok, gemv_rows;
    PyObject *dict, *qw, *gi, *perm;
    if (!PyArg_ParseTuple(args, "iiiiiOpiOOO", &K, &N, &bits, &group_size, &device, &dict, &gemm_ok, &gemv_rows, &qw, &gi, &perm))
        return nullptr;
    PyObject* buffers = PyDict_Check(dict) ? PyDict_GetItem(dict, s_buffers) : nullptr;
    if (!buffers) { PyErr_SetString(PyExc_TypeError, "module_dict"); return nullptr; }
    PyObject *pq = PyDict_GetItem(buffers, s_qweight), *pg = PyDict_GetItem(buffers, s_g_idx),
             *pz = PyDict_GetItem(buffers, s_qzeros), *ps = PyDict_GetItem(buffers, s_scales);
    PyObject* bias = PyDict_GetItem(buffers, s_bias);
    if (!bias) bias = PyDict_GetItem(dict, s_bias);
    PyObject* tuning = PyDict_GetItem(dict, s_gemv_tuning);
    if (!pq || !pg || !pz || !ps || !THPVariable_Check(pq) || !THPVariable_Check(pg) || !THPVariable_Check(pz) || !THPVariable_Check(ps) ||
        (bias && bias != Py_None && !THPVariable_Check(bias))) {
        PyErr_SetString(PyExc_TypeError, "the module lacks a buffer");
        return nullptr;
    }
    // (the stored qweight and g_idx too: as long as they live nothing else can come to lie at their addresses)
    PyObject* keep = PyTuple_Pack(9, pq, pg, qw, gi, perm, pz, ps, bias ? bias : Py_None, tuning ? tuning : Py_None);
    if (!keep) return nullptr;
    Layer* self = reinterpret_cast<Layer*>(type->tp_alloc(type, 0));
    if (!self) { Py_DECREF(keep); return nullptr; }
    self->K = K; self->N = N; self->bits = bits; self->group_size = group_size; self->device = device;
    self->writes = writes_to(pq) + writes_to(pg) + writes_to(pz) + writes_to(ps);
    self->qweight_at = tensor_address(pq);
    self->g_idx_at = tensor_address(pg);
    self->qzeros = pz; self->scales = ps; self->bias = bias ? bias : Py_None; self->tuning = tuning;
    self->gemm_ok = gemm_ok != 0;
    self->gemv_rows = gemv_rows < kMaxGemvRows ? gemv_rows : kMaxGemvRows;
    self->qweight_run = static_cast<const int32_t*>(tensor_address(qw));
    self->g_idx_run = static_cast<const int32_t*>(tensor_address(gi));
    self->x_perm = static_cast<const int32_t*>(tensor_address(perm));
    self->qzeros_run = static_cast<const int32_t*>(tensor_address(pz));
    self->scales_run = tensor_address(ps);
    self->bias_run = tensor_address(bias);
    self->keep = keep;
    return reinterpret_cast<PyObject*>(self);
}

PyObject* layer_new(PyTypeObject* type, PyObject* args, PyObject*) {
    try {
        return make_layer(type, args);
    } catch (const std::exception& e) {      // a tensor without an address
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

void layer_dealloc(PyObject* self_) {
    Layer* self = reinterpret_cast<Layer*>(self_);
    for (auto& e : self->gemv) Py_XDECREF(e.owner);
    Py_XDECREF(self->keep);
    Py_TYPE(self_)->tp_free(self_);
}

PyMethodDef layer_methods[] = {
    {"run", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(layer_run)), METH_FASTCALL, nullptr},
    {"set_gemv", layer_set_gemv, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyTypeObject LayerType = {PyVarObject_HEAD_INIT(nullptr, 0) "autogptq.tvm_b200._host.Layer", sizeof(Layer)};

// set_scratch(device, stream, tensor, bytes, in_graph)
PyObject* set_scratch(PyObject*, PyObject* args) {
    int device, in_graph;
    unsigned long long stream, bytes;
    PyObject* tensor;
    if (!PyArg_ParseTuple(args, "iKOKp", &device, &stream, &tensor, &bytes, &in_graph)) return nullptr;
    const void* address = nullptr;
    try {
        address = tensor_address(tensor);
    } catch (const std::exception&) {
    }
    if (!address) { PyErr_SetString(PyExc_TypeError, "set_scratch: a tensor"); return nullptr; }
    Scratch& s = (*g_scratch)[{device, (void*)(uintptr_t)stream}];
    PyObject* before = s.owner;
    Py_INCREF(tensor);
    s = Scratch{tensor, const_cast<void*>(address), (size_t)bytes, in_graph != 0};
    Py_XDECREF(before);
    Py_RETURN_NONE;
}
// scratch_use(device, stream): notes that the stream's scratch is handed out; (the stream is being captured, a graph may hold the
// address of the scratch)
PyObject* scratch_use(PyObject*, PyObject* args) {
    int device;
    unsigned long long stream;
    if (!PyArg_ParseTuple(args, "iK", &device, &stream)) return nullptr;
    bool capturing = false;
    try {
        capturing = is_capturing((cudaStream_t)(uintptr_t)stream);
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
    auto it = g_scratch->find({device, (void*)(uintptr_t)stream});
    if (it != g_scratch->end()) it->second.in_graph = it->second.in_graph || capturing;
    return Py_BuildValue("(NN)", PyBool_FromLong(capturing), PyBool_FromLong(it != g_scratch->end() && it->second.in_graph));
}
// zeros_outside_capture(device, bytes): zeroed memory that exists now, while a stream of this thread is being captured.  (An ordinary
// allocation would come from the graph's own memory, and be zeroed by the graph.)
PyObject* zeros_outside_capture(PyObject*, PyObject* args) {
    int device;
    long long bytes;
    if (!PyArg_ParseTuple(args, "iL", &device, &bytes)) return nullptr;
    try {
        const c10::cuda::CUDAGuard on((c10::DeviceIndex)device);
        const c10::cuda::CUDAStreamCaptureModeGuard relaxed{cudaStreamCaptureModeRelaxed};
        // (streams of the pool are handed out in turn: one of them may be the one that is captured)
        c10::cuda::CUDAStream side = c10::cuda::getStreamFromPool(false, (c10::DeviceIndex)device);
        for (int i = 0; i < 64 && is_capturing(side.stream()); ++i) side = c10::cuda::getStreamFromPool(false, (c10::DeviceIndex)device);
        const c10::cuda::CUDAStreamGuard beside(side);
        at::Tensor t = at::detail::empty_cuda({bytes}, at::kByte, at::Device(at::kCUDA, (c10::DeviceIndex)device), std::nullopt);
        C10_CUDA_CHECK(cudaMemsetAsync(t.mutable_data_ptr(), 0, (size_t)bytes, side.stream()));
        C10_CUDA_CHECK(cudaStreamSynchronize(side.stream()));
        return THPVariable_Wrap(std::move(t));
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}
// pack(weight, scales, zeros, g_idx, bits, copy_g_idx): QuantLinear.pack's (qweight, qzeros, scales, copy of g_idx or None) in one launch, or None
// where the Python route has more to do (another type, order, device or shape).
PyObject* pack_prepared(PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 6) { PyErr_SetString(PyExc_TypeError, "pack(weight, scales, zeros, g_idx, bits, copy_g_idx)"); return nullptr; }
    const at::Tensor* t[4];
    for (int i = 0; i < 4; ++i) {
        if (!THPVariable_Check(args[i])) Py_RETURN_NONE;
        t[i] = &THPVariable_Unpack(args[i]);
        if (t[i]->key_set().has_any(kNotPlain) || !t[i]->is_cuda() || !t[i]->is_contiguous()) Py_RETURN_NONE;
    }
    const at::Tensor &w = *t[0], &scales = *t[1], &zeros = *t[2], &g_idx = *t[3];
    const int bits = (int)PyLong_AsLong(args[4]), copy = PyObject_IsTrue(args[5]);
    if (PyErr_Occurred()) return nullptr;
    const auto type = w.scalar_type();
    const int dtype = type == at::kHalf ? B200GPTQ_F16 : (type == at::kBFloat16 ? B200GPTQ_BF16 : (type == at::kFloat ? B200GPTQ_F32 : -1));
    const int device = w.get_device();
    if (dtype < 0 || w.dim() != 2 || scales.dim() != 2 || scales.scalar_type() != at::kFloat || zeros.scalar_type() != at::kFloat ||
        g_idx.scalar_type() != at::kInt || g_idx.dim() != 1 || scales.get_device() != device || zeros.get_device() != device ||
        g_idx.get_device() != device || c10::cuda::current_device() != device)
        Py_RETURN_NONE;
    const int64_t N = w.size(0), K = w.size(1), G = scales.size(1);
    const void* wp = w.unsafeGetTensorImpl()->data();
    if (scales.size(0) != N || zeros.sizes() != scales.sizes() || g_idx.numel() != K || G < 1 || K < 32 || K % 32 || N < 32 || N % 32 ||
        K > INT32_MAX || N > INT32_MAX || ((uintptr_t)wp & 15u))
        Py_RETURN_NONE;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    const at::Device on(at::kCUDA, (c10::DeviceIndex)device);
    at::Tensor qweight, qzeros, scales16, g_copy;
    int st;
    {
        const WithoutGil released;
        qweight = at::detail::empty_cuda({K / 32 * bits, N}, at::kInt, on, std::nullopt);
        qzeros = at::detail::empty_cuda({G, N / 32 * bits}, at::kInt, on, std::nullopt);
        scales16 = at::detail::empty_cuda({G, N}, at::kHalf, on, std::nullopt);
        if (copy) g_copy = at::detail::empty_cuda({K}, at::kInt, on, std::nullopt);
        auto ints = [](at::Tensor& x) { return static_cast<int32_t*>(x.unsafeGetTensorImpl()->mutable_data()); };
        st = b200gptq_pack_linear_ex(wp, dtype, static_cast<const float*>(scales.unsafeGetTensorImpl()->data()),
                                     static_cast<const float*>(zeros.unsafeGetTensorImpl()->data()),
                                     static_cast<const int32_t*>(g_idx.unsafeGetTensorImpl()->data()), (int)K, (int)N, (int)G, bits,
                                     ints(qweight), ints(qzeros), scales16.unsafeGetTensorImpl()->mutable_data(),
                                     copy ? ints(g_copy) : nullptr, stream);
    }
    if (st != B200GPTQ_OK) Py_RETURN_NONE;   // the Python route repeats the call and reports the status
    PyObject* out[4] = {THPVariable_Wrap(std::move(qweight)), THPVariable_Wrap(std::move(qzeros)), THPVariable_Wrap(std::move(scales16)),
                        copy ? THPVariable_Wrap(std::move(g_copy)) : Py_NewRef(Py_None)};
    return Py_BuildValue("(NNNN)", out[0], out[1], out[2], out[3]);
}
PyObject* pack(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    try {
        return pack_prepared(args, nargs);
    } catch (const std::exception&) {        // out of memory: met again by the Python route, which raises it with its own type
        Py_RETURN_NONE;
    }
}
PyObject* set_scratch_source(PyObject*, PyObject* fn) {
    Py_INCREF(fn);
    Py_XSETREF(g_get_workspace, fn);
    Py_RETURN_NONE;
}

PyMethodDef module_methods[] = {
    {"pack", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(pack)), METH_FASTCALL, nullptr},
    {"set_scratch", set_scratch, METH_VARARGS, nullptr},
    {"set_scratch_source", set_scratch_source, METH_O, nullptr},
    {"scratch_use", scratch_use, METH_VARARGS, nullptr},
    {"zeros_outside_capture", zeros_outside_capture, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, module_methods};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    g_scratch = new std::unordered_map<std::pair<int, void*>, Scratch, KeyHash>();
    s_buffers = PyUnicode_InternFromString("_buffers");
    s_qweight = PyUnicode_InternFromString("qweight");
    s_g_idx = PyUnicode_InternFromString("g_idx");
    s_qzeros = PyUnicode_InternFromString("qzeros");
    s_scales = PyUnicode_InternFromString("scales");
    s_bias = PyUnicode_InternFromString("bias");
    s_gemv_tuning = PyUnicode_InternFromString("gemv_tuning");
    LayerType.tp_flags = Py_TPFLAGS_DEFAULT;
    LayerType.tp_new = layer_new;
    LayerType.tp_dealloc = layer_dealloc;
    LayerType.tp_methods = layer_methods;
    if (PyType_Ready(&LayerType) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&LayerType);
    if (PyModule_AddObject(m, "Layer", reinterpret_cast<PyObject*>(&LayerType)) < 0) return nullptr;
    return m;
}
