// Native call path of the Python layer (module turboquant_b200._native).
//
// A decode step's GPU work is a few microseconds per layer at short contexts, and a call through Python attribute
// checks and ctypes argument boxing cost 14 us (write) to 20 us (decode) of host time, which bounded every step below
// about 8 MB of cache.  Here a call takes its torch tensors as they are, checks shapes, types and devices in C++ and
// enters the C ABI: about a microsecond on top of the kernel launches.
//
// The entry points of the C ABI come as addresses from the ctypes handle (bind), so there is one library and one
// override of its path.  Every call here has the answer "not mine" (Python None): anything but the plain case - an
// output that must be viewed, an int64 table, a first call whose workspace does not exist yet, TQ_DEBUG_CHECKS - goes
// back to the Python layer, which converts, allocates or raises with its message, and calls the same entry point.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <unordered_map>

#include "../../include/turboquant_b200.h"

namespace {

decltype(&tq_write_kv_cache) fn_write = nullptr;
decltype(&tq_decode_paged_multi) fn_multi = nullptr;
decltype(&tq_decode_paged_causal) fn_causal = nullptr;
decltype(&tq_dequant_paged) fn_dequant = nullptr;
decltype(&tq_quantize_flat) fn_quantize = nullptr;
decltype(&tq_dequantize_flat) fn_dequantize = nullptr;
decltype(&tq_last_error) fn_last_error = nullptr;
PyObject* error_class = nullptr;

constexpr int kMaxDevices = 64;

struct Gil {  // the launches run without the interpreter lock, as a ctypes call does
    PyThreadState* state = PyEval_SaveThread();
    ~Gil() { PyEval_RestoreThread(state); }
};

bool debug_checks() {
    const char* v = std::getenv("TQ_DEBUG_CHECKS");
    return v && *v && !(v[0] == '0' && v[1] == 0);
}

const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
const at::Tensor* cuda_tensor(PyObject* o) {
    const at::Tensor* t = tensor(o);
    return t && t->is_cuda() && t->layout() == at::kStrided && t->get_device() < kMaxDevices ? t : nullptr;
}
int float_code(at::ScalarType t) {
    return t == at::kFloat ? TQ_F32 : t == at::kHalf ? TQ_F16 : t == at::kBFloat16 ? TQ_BF16 : -1;
}
bool int32_table(const at::Tensor* t, int device) {
    return t && t->get_device() == device && t->scalar_type() == at::kInt && t->is_contiguous();
}
bool byte_cache(const at::Tensor* t) {
    return t && t->dim() == 5 && t->size(0) == 2 && t->is_contiguous() && t->element_size() == 1;
}
void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

PyObject* failed(int rc) {
    return PyErr_Format(error_class, "turboquant_b200 error %d: %s", rc, fn_last_error());
}

// -------------------------------------------------------------------------------------------------
// Layer: one attention geometry with its sign vectors and workspaces (the Python object hands them over)
// -------------------------------------------------------------------------------------------------
struct Layer {
    PyObject_HEAD
    int heads, head_size, kv_heads, num_ctas;
    float scale;
    at::Tensor* signs;                                      // [kMaxDevices]
    std::unordered_map<uint64_t, at::Tensor>* workspaces;   // (device, queries, batch)
};

uint64_t ws_key(int device, int64_t batch, int64_t queries) {
    return (uint64_t)device << 56 | (uint64_t)(queries & 0xffffff) << 32 | (uint64_t)(uint32_t)batch;
}

PyObject* layer_new(PyTypeObject* type, PyObject* args, PyObject*) {
    int heads, head_size, kv_heads, num_ctas;
    float scale;
    if (!PyArg_ParseTuple(args, "iiifi", &heads, &head_size, &kv_heads, &scale, &num_ctas)) return nullptr;
    Layer* self = reinterpret_cast<Layer*>(type->tp_alloc(type, 0));
    if (!self) return nullptr;
    self->heads = heads;
    self->head_size = head_size;
    self->kv_heads = kv_heads;
    self->num_ctas = num_ctas;
    self->scale = scale;
    self->signs = new at::Tensor[kMaxDevices];
    self->workspaces = new std::unordered_map<uint64_t, at::Tensor>();
    return reinterpret_cast<PyObject*>(self);
}

void layer_dealloc(PyObject* o) {
    Layer* self = reinterpret_cast<Layer*>(o);
    delete[] self->signs;
    delete self->workspaces;
    PyTypeObject* type = Py_TYPE(o);
    type->tp_free(o);
    Py_DECREF(type);
}

// set_signs(tensor), set_workspace(batch, queries, tensor)
PyObject* layer_set_signs(PyObject* o, PyObject* arg) {
    HANDLE_TH_ERRORS
    const at::Tensor* t = cuda_tensor(arg);
    if (t && t->scalar_type() == at::kFloat && t->is_contiguous()) reinterpret_cast<Layer*>(o)->signs[t->get_device()] = *t;
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}
PyObject* layer_set_workspace(PyObject* o, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const at::Tensor* t = n == 3 ? cuda_tensor(args[2]) : nullptr;
    if (t) {
        const int64_t batch = PyLong_AsLongLong(args[0]), queries = PyLong_AsLongLong(args[1]);
        if (PyErr_Occurred()) return nullptr;
        (*reinterpret_cast<Layer*>(o)->workspaces)[ws_key(t->get_device(), batch, queries)] = *t;
    }
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// write(key, value, kv_cache, slot_mapping, zero_pad) -> True, or None: not the plain case
PyObject* layer_write(PyObject* o, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Layer* self = reinterpret_cast<Layer*>(o);
    if (n != 5 || debug_checks()) Py_RETURN_NONE;
    const at::Tensor *k = cuda_tensor(args[0]), *v = cuda_tensor(args[1]), *cache = cuda_tensor(args[2]), *slots = cuda_tensor(args[3]);
    if (!k || !v || !slots || !byte_cache(cache)) Py_RETURN_NONE;
    const int dev = cache->get_device(), dtype = float_code(k->scalar_type());
    const at::Tensor& signs = self->signs[dev];
    if (!signs.defined() || dtype < 0 || k->get_device() != dev || v->get_device() != dev || slots->get_device() != dev) Py_RETURN_NONE;
    const int64_t H = self->kv_heads, D = self->head_size, T = slots->size(0);
    if (slots->dim() != 1 || !slots->is_contiguous() || (slots->scalar_type() != at::kLong && slots->scalar_type() != at::kInt)) Py_RETURN_NONE;
    if (cache->size(3) != H || v->scalar_type() != k->scalar_type()) Py_RETURN_NONE;
    for (const at::Tensor* t : {k, v})
        if (t->dim() != 3 || t->size(0) < T || t->size(1) != H || t->size(2) != D || t->stride(2) != 1 || t->stride(1) != D) Py_RETURN_NONE;
    if (T == 0) Py_RETURN_TRUE;
    const int zero_pad = PyObject_IsTrue(args[4]);
    if (zero_pad < 0) return nullptr;
    void* stream = stream_of(dev);
    int rc;
    {
        Gil gil;
        rc = fn_write(cache->data_ptr(), cache->size(1), (int)cache->size(2), (int)H, (int)cache->size(4), k->data_ptr(), v->data_ptr(),
                      dtype, T, k->stride(0), v->stride(0), static_cast<const float*>(signs.data_ptr()), slots->data_ptr(),
                      slots->scalar_type() == at::kLong ? TQ_I64 : TQ_I32, (int)D, zero_pad ? TQ_WRITE_ZERO_PAD : TQ_WRITE_DEFAULT, stream);
    }
    if (rc) return failed(rc);
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// decode(query, kv_cache, block_table, seq_lens, output | None, out_lse | None, causal) -> output, or None: not the
// plain case.  query [batch, heads, size] (one query a row) or [batch, queries, heads, size].
PyObject* layer_decode(PyObject* o, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Layer* self = reinterpret_cast<Layer*>(o);
    if (n != 7 || debug_checks()) Py_RETURN_NONE;
    const at::Tensor *q = cuda_tensor(args[0]), *cache = cuda_tensor(args[1]), *table = cuda_tensor(args[2]), *lens = cuda_tensor(args[3]);
    if (!q || !byte_cache(cache)) Py_RETURN_NONE;
    const int dev = cache->get_device(), q_dtype = float_code(q->scalar_type());
    const int dims = (int)q->dim();
    if (dims < 3 || dims > 4 || q->get_device() != dev || q_dtype < 0 || !q->is_contiguous()) Py_RETURN_NONE;
    const int64_t B = q->size(0), NQ = dims == 4 ? q->size(1) : 1;
    if (q->size(dims - 2) != self->heads || q->size(dims - 1) != self->head_size || cache->size(3) != self->kv_heads) Py_RETURN_NONE;
    if (!int32_table(table, dev) || table->dim() < 1 || !int32_table(lens, dev) || lens->dim() != 1 || lens->size(0) != B) Py_RETURN_NONE;
    const at::Tensor& signs = self->signs[dev];
    const auto ws = self->workspaces->find(ws_key(dev, B, NQ));
    if (!signs.defined() || ws == self->workspaces->end()) Py_RETURN_NONE;
    float* lse = nullptr;
    if (args[5] != Py_None) {
        const at::Tensor* t = cuda_tensor(args[5]);
        if (!t || t->get_device() != dev || t->scalar_type() != at::kFloat || !t->is_contiguous() || t->numel() != B * NQ * self->heads) Py_RETURN_NONE;
        lse = static_cast<float*>(t->data_ptr());
    }
    at::Tensor fresh;
    const at::Tensor* out;
    if (args[4] == Py_None) {
        fresh = at::empty_like(*q);
        out = &fresh;
    } else {
        out = cuda_tensor(args[4]);
        if (!out || out->get_device() != dev || float_code(out->scalar_type()) < 0 || !out->is_contiguous() || out->numel() != q->numel()) Py_RETURN_NONE;
    }
    if (B > 0 && NQ > 0) {
        const size_t ws_bytes = ws->second.numel() * ws->second.element_size();
        void *ws_ptr = ws->second.data_ptr(), *stream = stream_of(dev);
        const float* sg = static_cast<const float*>(signs.data_ptr());
        const int out_dtype = float_code(out->scalar_type()), max_pages = (int)table->size(-1);
        const int32_t *pages = static_cast<const int32_t*>(table->data_ptr()), *sl = static_cast<const int32_t*>(lens->data_ptr());
        const bool causal = args[6] == Py_True;
        int rc;
        {
            Gil gil;
            rc = causal ? fn_causal(q->data_ptr(), q_dtype, (int)B, (int)NQ, self->heads, self->kv_heads, self->head_size, cache->data_ptr(),
                                    cache->size(1), (int)cache->size(2), (int)cache->size(4), pages, nullptr, max_pages, sl, sg, self->scale,
                                    ws_ptr, ws_bytes, out->data_ptr(), out_dtype, lse, self->num_ctas, stream)
                        : fn_multi(q->data_ptr(), q_dtype, (int)B, (int)NQ, self->heads, self->kv_heads, self->head_size, cache->data_ptr(),
                                   cache->size(1), (int)cache->size(2), (int)cache->size(4), pages, nullptr, max_pages, sl, 0, -1, sg,
                                   self->scale, ws_ptr, ws_bytes, out->data_ptr(), out_dtype, lse, 0, self->num_ctas, stream);
        }
        if (rc) return failed(rc);
    }
    if (fresh.defined()) return THPVariable_Wrap(std::move(fresh));
    return Py_NewRef(args[4]);
    END_HANDLE_TH_ERRORS
}

// dequant(kv_cache, block_table, seq_lens, cu_seqlens, total_tokens, dtype) -> (k, v), or None: not the plain case
PyObject* layer_dequant(PyObject* o, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Layer* self = reinterpret_cast<Layer*>(o);
    if (n != 6 || !THPDtype_Check(args[5]) || !PyLong_Check(args[4])) Py_RETURN_NONE;
    const at::Tensor *cache = cuda_tensor(args[0]), *table = cuda_tensor(args[1]), *lens = cuda_tensor(args[2]), *cu = cuda_tensor(args[3]);
    if (!byte_cache(cache)) Py_RETURN_NONE;
    const int dev = cache->get_device();
    const at::ScalarType type = reinterpret_cast<THPDtype*>(args[5])->scalar_type;
    const long long total = PyLong_AsLongLong(args[4]);
    if (total < 0 && PyErr_Occurred()) return nullptr;
    const at::Tensor& signs = self->signs[dev];
    if (!signs.defined() || float_code(type) < 0 || total <= 0 || cache->size(3) != self->kv_heads) Py_RETURN_NONE;
    if (!int32_table(table, dev) || table->dim() < 1 || !int32_table(lens, dev) || lens->dim() != 1 || !int32_table(cu, dev) ||
        cu->dim() != 1 || cu->size(0) != lens->size(0) + 1)
        Py_RETURN_NONE;
    const auto options = at::TensorOptions().dtype(type).device(cache->device());
    at::Tensor k = at::empty({total, self->kv_heads, self->head_size}, options), v = at::empty({total, self->kv_heads, self->head_size}, options);
    void* stream = stream_of(dev);
    int rc;
    {
        Gil gil;
        rc = fn_dequant(cache->data_ptr(), cache->size(1), (int)cache->size(2), (int)cache->size(3), (int)cache->size(4),
                        static_cast<const int32_t*>(table->data_ptr()), nullptr, (int)table->size(-1),
                        static_cast<const int32_t*>(lens->data_ptr()), static_cast<const int32_t*>(cu->data_ptr()), (int)lens->size(0),
                        static_cast<const float*>(signs.data_ptr()), self->head_size, k.data_ptr(), v.data_ptr(), float_code(type),
                        k.stride(0), stream);
    }
    if (rc) return failed(rc);
    PyObject *a = THPVariable_Wrap(std::move(k)), *b = THPVariable_Wrap(std::move(v));
    PyObject* pair = a && b ? PyTuple_Pack(2, a, b) : nullptr;
    Py_XDECREF(a);
    Py_XDECREF(b);
    return pair;
    END_HANDLE_TH_ERRORS
}

// -------------------------------------------------------------------------------------------------
// flat quantizer
// -------------------------------------------------------------------------------------------------
int64_t padded_dim(int64_t d) {
    int64_t p = 1;
    while (p < d) p <<= 1;
    return p;
}

// quantize_flat(x, signs, bits, cache_order) -> (packed, norms), or None
PyObject* quantize_flat(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const at::Tensor *x = n == 4 ? cuda_tensor(args[0]) : nullptr, *signs = n == 4 ? cuda_tensor(args[1]) : nullptr;
    if (!x || !signs || x->dim() < 1 || !x->is_contiguous() || x->numel() == 0 || float_code(x->scalar_type()) < 0) Py_RETURN_NONE;
    const long bits = PyLong_AsLong(args[2]);
    if (bits == -1 && PyErr_Occurred()) return nullptr;
    const int order = PyObject_IsTrue(args[3]);      // any truth value, as the Python layer takes it
    if (order < 0) return nullptr;
    const int64_t d = x->size(-1), pd = padded_dim(d);
    if (bits < 1 || bits > 4 || signs->get_device() != x->get_device() || signs->scalar_type() != at::kFloat || !signs->is_contiguous() ||
        signs->numel() < pd)
        Py_RETURN_NONE;
    const int64_t rows = x->numel() / d, per = 8 / bits;
    const auto options = at::TensorOptions().device(x->device());
    at::DimVector shape(x->sizes());
    shape.back() = (pd + per - 1) / per;
    at::Tensor packed = at::empty(shape, options.dtype(at::kByte));
    shape.pop_back();
    at::Tensor norms = at::empty(shape, options.dtype(at::kFloat));
    void* stream = stream_of(x->get_device());
    int rc;
    {
        Gil gil;
        rc = fn_quantize(x->data_ptr(), float_code(x->scalar_type()), rows, (int)d, static_cast<const float*>(signs->data_ptr()), (int)bits,
                         order ? TQ_PACK_CACHE : TQ_PACK_LOW_FIRST, static_cast<uint8_t*>(packed.data_ptr()),
                         static_cast<float*>(norms.data_ptr()), stream);
    }
    if (rc) return failed(rc);
    PyObject *a = THPVariable_Wrap(std::move(packed)), *b = THPVariable_Wrap(std::move(norms));
    PyObject* pair = a && b ? PyTuple_Pack(2, a, b) : nullptr;
    Py_XDECREF(a);
    Py_XDECREF(b);
    return pair;
    END_HANDLE_TH_ERRORS
}

// dequantize_flat(packed, norms, signs, dim, bits, cache_order) -> x, or None
PyObject* dequantize_flat(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 6) Py_RETURN_NONE;
    const at::Tensor *packed = cuda_tensor(args[0]), *norms = cuda_tensor(args[1]), *signs = cuda_tensor(args[2]);
    if (!packed || !norms || !signs || packed->dim() < 1) Py_RETURN_NONE;
    const long d = PyLong_AsLong(args[3]), bits = PyLong_AsLong(args[4]);
    const int order = PyErr_Occurred() ? -1 : PyObject_IsTrue(args[5]);
    if (order < 0) return nullptr;
    const int dev = packed->get_device();
    if (norms->get_device() != dev || signs->get_device() != dev || packed->scalar_type() != at::kByte || !packed->is_contiguous() ||
        norms->scalar_type() != at::kFloat || !norms->is_contiguous() || signs->scalar_type() != at::kFloat || !signs->is_contiguous())
        Py_RETURN_NONE;
    if (d < 1 || bits < 1 || bits > 4) Py_RETURN_NONE;
    const int64_t rows = norms->numel(), pd = padded_dim(d), per = 8 / bits;
    if (rows == 0 || packed->numel() != rows * ((pd + per - 1) / per) || signs->numel() < pd) Py_RETURN_NONE;
    at::DimVector shape(norms->sizes());
    shape.push_back(d);
    at::Tensor out = at::empty(shape, at::TensorOptions().device(packed->device()).dtype(at::kFloat));
    void* stream = stream_of(dev);
    int rc;
    {
        Gil gil;
        rc = fn_dequantize(static_cast<const uint8_t*>(packed->data_ptr()), static_cast<const float*>(norms->data_ptr()), rows, (int)d,
                           static_cast<const float*>(signs->data_ptr()), (int)bits, order ? TQ_PACK_CACHE : TQ_PACK_LOW_FIRST,
                           static_cast<float*>(out.data_ptr()), stream);
    }
    if (rc) return failed(rc);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// bind(addresses: dict name -> int, error class)
PyObject* bind(PyObject*, PyObject* args) {
    PyObject *table, *cls;
    if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &table, &cls)) return nullptr;
    auto take = [&](const char* name, auto& fn) {
        PyObject* v = PyDict_GetItemString(table, name);
        void* p = v ? PyLong_AsVoidPtr(v) : nullptr;
        fn = reinterpret_cast<std::decay_t<decltype(fn)>>(p);
        return p != nullptr;
    };
    if (!take("tq_write_kv_cache", fn_write) || !take("tq_decode_paged_multi", fn_multi) || !take("tq_decode_paged_causal", fn_causal) ||
        !take("tq_dequant_paged", fn_dequant) || !take("tq_quantize_flat", fn_quantize) || !take("tq_dequantize_flat", fn_dequantize) ||
        !take("tq_last_error", fn_last_error)) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "bind: an entry point is missing");
        return nullptr;
    }
    Py_XSETREF(error_class, Py_NewRef(cls));
    Py_RETURN_NONE;
}

PyMethodDef layer_methods[] = {
    {"set_signs", layer_set_signs, METH_O, nullptr},
    {"set_workspace", (PyCFunction)(void (*)())layer_set_workspace, METH_FASTCALL, nullptr},
    {"write", (PyCFunction)(void (*)())layer_write, METH_FASTCALL, nullptr},
    {"decode", (PyCFunction)(void (*)())layer_decode, METH_FASTCALL, nullptr},
    {"dequant", (PyCFunction)(void (*)())layer_dequant, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyType_Slot layer_slots[] = {{Py_tp_new, (void*)layer_new}, {Py_tp_dealloc, (void*)layer_dealloc}, {Py_tp_methods, layer_methods}, {0, nullptr}};
PyType_Spec layer_spec = {"turboquant_b200._native.Layer", sizeof(Layer), 0, Py_TPFLAGS_DEFAULT, layer_slots};

PyMethodDef module_methods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"quantize_flat", (PyCFunction)(void (*)())quantize_flat, METH_FASTCALL, nullptr},
    {"dequantize_flat", (PyCFunction)(void (*)())dequantize_flat, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    PyObject* type = PyType_FromSpec(&layer_spec);
    if (!type || PyModule_AddObject(m, "Layer", type) < 0) return nullptr;
    return m;
}
