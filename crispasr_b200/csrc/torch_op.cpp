// torch_op.cpp — the Python call surface of op.py in native code: torch tensors to b200_tensor descriptors, output and
// workspace from torch's caching allocator, one planned launch through the C-ABI.
//
// A decode step of a small model is a few launches of 4-8 us each, so what a call costs on the host decides the step:
// the same work in Python (about sixty attribute reads and ctypes objects per call, the operator planned twice) took
// 27-33 us per call, this module 4 us, most of it the kernel launch and the output allocation.  A 6-layer step of Whisper
// base.en (12 calls) 400 -> 58 us and, as vector calls without a Python function in front, 54 us; a 30-layer Q8_0 decoder
// step (60 calls) 1604 -> 492 us before its kernels became faster.
#include <Python.h>

#include <exception>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200_fattn.h"

namespace {

// Interned names of the arguments, compared by pointer first (keyword names of call sites are interned).
enum Key { kScale, kMaxBias, kSoftcap, kKvType, kCausal, kNPast, kKvLen, kQv, kR, kRelposF32, kBiasU, kBiasV, kKvIndex, kQLen, kOut,
           kWorkspace, kStream, kQ, kK, kV, kMask, kKeys };
const char* const kKeyNames[kKeys] = {"scale", "max_bias", "softcap", "kv_type", "causal", "n_past", "kv_len", "q_v", "r",
                                      "relpos_bias_f32", "pos_bias_u", "pos_bias_v", "kv_index", "q_len", "out", "workspace", "stream",
                                      "q", "k", "v", "mask"};
PyObject* g_keys[kKeys];

struct Kwargs {
    PyObject* v[kKeys] = {};   // borrowed; null = absent, or None where that is a value (a number has to be one)
    // `values`: those of the keyword names, behind the positional arguments of a vector call
    bool parse(PyObject* names, PyObject* const* values) {
        const Py_ssize_t n = names ? PyTuple_GET_SIZE(names) : 0;
        for (Py_ssize_t j = 0; j < n; j++) {
            PyObject* name = PyTuple_GET_ITEM(names, j);
            int hit = -1;
            for (int i = 0; i < kKeys && hit < 0; i++)
                if (name == g_keys[i]) hit = i;
            for (int i = 0; i < kKeys && hit < 0; i++)
                if (PyUnicode_Compare(name, g_keys[i]) == 0) hit = i;
            if (PyErr_Occurred()) return false;
            const bool number = hit == kScale || hit == kMaxBias || hit == kSoftcap || hit == kNPast;
            if (hit >= 0) v[hit] = values[j] == Py_None && !number ? nullptr : values[j];   // other names are ignored, as they always were
        }
        return true;
    }
    // q, k, v, mask: by position or by name
    bool operands(PyObject* const* a, Py_ssize_t n, const char* where, PyObject* (&op)[4]) const {
        if (n > 4) {
            PyErr_Format(PyExc_TypeError, "%s() takes from 3 to 4 positional arguments but %zd were given", where, n);
            return false;
        }
        for (int i = 0; i < 4; i++) {
            if (i < n && v[kQ + i]) {
                PyErr_Format(PyExc_TypeError, "%s() got multiple values for argument '%s'", where, kKeyNames[kQ + i]);
                return false;
            }
            op[i] = i < n ? a[i] : v[kQ + i];
            if (!op[i] && i < 3) {
                PyErr_Format(PyExc_TypeError, "%s() missing required argument '%s'", where, kKeyNames[kQ + i]);
                return false;
            }
        }
        return true;
    }
    bool number(Key k, double dflt, double* out) const {
        if (!v[k]) return *out = dflt, true;
        PyObject* f = PyNumber_Float(v[k]);   // float(x): texts as well
        if (!f) return false;
        *out = PyFloat_AS_DOUBLE(f);
        Py_DECREF(f);
        return true;
    }
    bool integer(Key k, long* out) const {
        if (!v[k]) return *out = 0, true;
        PyObject* i = PyNumber_Long(v[k]);
        if (!i) return false;
        *out = PyLong_AsLong(i);
        Py_DECREF(i);
        return !(*out == -1 && PyErr_Occurred());
    }
    bool truth(Key k, int32_t* out) const {
        const int t = v[k] ? PyObject_IsTrue(v[k]) : 0;
        *out = t;
        return t >= 0;
    }
};

const at::Tensor* tensor_of(PyObject* o, const char* what) {
    if (THPVariable_Check(o)) return &THPVariable_Unpack(o);
    PyErr_Format(PyExc_TypeError, "%s is a torch tensor, not %s", what, Py_TYPE(o)->tp_name);
    return nullptr;
}

// torch order (slowest first) -> ggml order; absent dimensions get the strides of the full extent.
bool describe(const at::Tensor& x, long type, b200_tensor* t) {
    const auto st = x.scalar_type();
    if (type < 0) {
        if (st == at::kFloat) type = B200_TYPE_F32;
        else if (st == at::kHalf) type = B200_TYPE_F16;
        else {
            PyErr_Format(PyExc_KeyError, "torch.%s", c10::toString(st));
            return false;
        }
    }
    const int nd = (int)x.dim();
    if (nd > 4) {
        PyErr_SetString(PyExc_ValueError, "at most 4 dimensions");
        return false;
    }
    const bool q8 = type == B200_TYPE_Q8_0;
    if (q8 && (st != at::kByte || nd == 0 || x.stride(-1) != 1)) {
        PyErr_SetString(PyExc_ValueError, "Q8_0 tensors are uint8 with a contiguous last axis");
        return false;
    }
    const int64_t es = x.element_size();
    t->data = x.data_ptr();
    t->type = (int32_t)type;
    t->reserved = 0;
    for (int i = 0; i < 4; i++) t->ne[i] = 1, t->nb[i] = 0;
    for (int i = 0; i < nd; i++) {
        t->ne[i] = x.size(nd - 1 - i);
        t->nb[i] = (uint64_t)(x.stride(nd - 1 - i) * es);
    }
    if (q8) t->ne[0] = t->ne[0] / 34 * 32, t->nb[0] = 34;
    if (nd == 0) t->nb[0] = (uint64_t)es;
    for (int i = nd > 1 ? nd : 1; i < 4; i++) t->nb[i] = t->nb[i - 1] * (uint64_t)(q8 && i == 1 ? t->ne[0] / 32 : t->ne[i - 1]);
    return true;
}

// Address of an index table: a torch tensor's, that of any other object with data_ptr(), or a numpy array's.
bool address_of(PyObject* o, const int32_t** out) {
    if (THPVariable_Check(o)) {
        *out = (const int32_t*)THPVariable_Unpack(o).data_ptr();
        return true;
    }
    PyObject* data = nullptr;
    if (PyObject_HasAttrString(o, "data_ptr")) {
        data = PyObject_CallMethod(o, "data_ptr", nullptr);
    } else {
        PyObject* ct = PyObject_GetAttrString(o, "ctypes");
        data = ct ? PyObject_GetAttrString(ct, "data") : nullptr;
        Py_XDECREF(ct);
    }
    if (!data) return false;
    *out = (const int32_t*)PyLong_AsVoidPtr(data);
    Py_DECREF(data);
    return !PyErr_Occurred();
}

bool last_extent(PyObject* o, int32_t* out) {
    if (THPVariable_Check(o)) {
        *out = (int32_t)THPVariable_Unpack(o).size(-1);
        return true;
    }
    PyObject* shape = PyObject_GetAttrString(o, "shape");
    const Py_ssize_t n = shape ? PySequence_Length(shape) : -1;
    PyObject* last = n > 0 ? PySequence_GetItem(shape, n - 1) : nullptr;
    Py_XDECREF(shape);
    if (!last) return false;
    *out = (int32_t)PyLong_AsLong(last);
    Py_DECREF(last);
    return !PyErr_Occurred();
}

// Stream handle: None (the caller picks), an integer, a ctypes pointer, or an object that has one for ctypes (`_as_parameter_`:
// torch.cuda.Stream).
bool stream_of(PyObject* o, void** out) {
    if (PyLong_Check(o)) {
        *out = PyLong_AsVoidPtr(o);
        return !PyErr_Occurred();
    }
    if (PyObject* as = PyObject_GetAttrString(o, "_as_parameter_")) {
        const bool ok = PyLong_Check(as) || PyObject_HasAttrString(as, "value");
        if (!ok) PyErr_SetString(PyExc_TypeError, "stream is an integer, a ctypes pointer or a torch.cuda.Stream");
        const bool got = ok && stream_of(as, out);
        Py_DECREF(as);
        return got;
    }
    PyErr_Clear();
    PyObject* value = PyObject_GetAttrString(o, "value");
    if (!value) return false;
    *out = value == Py_None ? nullptr : PyLong_AsVoidPtr(value);
    Py_DECREF(value);
    return !PyErr_Occurred();
}

PyObject* raise_code(int rc, const char* where) {
    PyObject* mod = PyImport_ImportModule("crispasr_b200");
    PyObject* cls = mod ? PyObject_GetAttrString(mod, "B200Error") : nullptr;
    PyObject* err = cls ? PyObject_CallFunction(cls, "is", rc, where) : nullptr;
    if (err) PyErr_SetObject(cls, err);
    Py_XDECREF(err);
    Py_XDECREF(cls);
    Py_XDECREF(mod);
    return nullptr;
}

struct Operands {
    b200_tensor q, k, v, mask, dst, qv, r, bu, bv;
    bool has_mask = false;
    b200_fattn_params params;
    b200_fattn_ext ext;
    const b200_tensor* mask_p() const { return has_mask ? &mask : nullptr; }

    bool fill(PyObject* q_, PyObject* k_, PyObject* v_, PyObject* mask_, const Kwargs& kw) {
        if (!kw.v[kScale]) {
            PyErr_SetString(PyExc_KeyError, "scale");
            return false;
        }
        long kv_type = -1, n_past = 0;
        if (kw.v[kKvType] && !kw.integer(kKvType, &kv_type)) return false;
        const at::Tensor *tk = tensor_of(k_, "k"), *tv = tk ? tensor_of(v_, "v") : nullptr;
        if (!tv || !describe(THPVariable_Unpack(q_), -1, &q) || !describe(*tk, kv_type, &k) || !describe(*tv, kv_type, &v)) return false;
        if (mask_ && mask_ != Py_None) {
            const at::Tensor* tm = tensor_of(mask_, "mask");
            if (!tm || !describe(*tm, -1, &mask)) return false;
            has_mask = true;
        }
        double scale, max_bias, softcap;
        if (!kw.number(kScale, 0.0, &scale) || !kw.number(kMaxBias, 0.0, &max_bias) || !kw.number(kSoftcap, 0.0, &softcap)) return false;
        params = b200_fattn_params{(float)scale, (float)max_bias, (float)softcap, 0};
        ext = b200_fattn_ext{};
        const struct { Key key; b200_tensor* t; const b200_tensor** slot; const char* name; } opt[4] = {
            {kQv, &qv, &ext.q_v, "q_v"}, {kR, &r, &ext.r, "r"}, {kBiasU, &bu, &ext.pos_bias_u, "pos_bias_u"}, {kBiasV, &bv, &ext.pos_bias_v, "pos_bias_v"}};
        for (const auto& o : opt)
            if (kw.v[o.key]) {
                const at::Tensor* t = tensor_of(kw.v[o.key], o.name);
                if (!t || !describe(*t, -1, o.t)) return false;
                *o.slot = o.t;
            }
        if (!kw.truth(kCausal, &ext.causal) || !kw.integer(kNPast, &n_past) || !kw.truth(kRelposF32, &ext.relpos_bias_f32)) return false;
        ext.n_past = (int32_t)n_past;
        if (kw.v[kKvLen] && !address_of(kw.v[kKvLen], &ext.kv_len)) return false;
        if (kw.v[kKvIndex] && (!address_of(kw.v[kKvIndex], &ext.kv_index) || !last_extent(kw.v[kKvIndex], &ext.kv_index_stride))) return false;
        return !kw.v[kQLen] || address_of(kw.v[kQLen], &ext.q_len);
    }
};

struct Scratch {
    at::Tensor buf;
    c10::Device device;
    void* given;
    size_t given_bytes;
    void* stream;   // the launch's
    std::exception_ptr error;   // what the allocator raised: it must not pass through the C entry point, the caller gets it behind that
};
void* scratch_alloc(void* user, size_t bytes) {
    Scratch* s = (Scratch*)user;
    if (s->given && s->given_bytes >= bytes) return s->given;
    try {
        // The block comes from the pool of the stream that uses it: one of the current stream's pool may still be in use by
        // that stream's earlier work, and would be handed out again while this launch is in flight.
        c10::cuda::OptionalCUDAStreamGuard on_stream;
        const cudaStream_t st = s->stream == (void*)cudaStreamLegacy ? nullptr : (cudaStream_t)s->stream;
        if (st != c10::cuda::getCurrentCUDAStream(s->device.index()).stream())
            on_stream.reset_stream(c10::cuda::getStreamFromExternal(st, s->device.index()));
        s->buf = at::detail::empty_cuda({(int64_t)bytes}, at::kByte, s->device, std::nullopt);
    } catch (...) {
        s->error = std::current_exception();
        return nullptr;
    }
    return s->buf.data_ptr();
}

const char kLaunchDoc[] =
    "flash_attn_ext(q, k, v, mask=None, *, out=None, workspace=None, stream=None, **kw)\n--\n\n"
    "Device tensors in, device tensor out; asynchronous on `stream` (default: torch's current stream).\n"
    "`workspace` (uint8 device tensor) is allocated here, for `stream`, when the launch needs one and none is given; the\n"
    "result comes from the current stream's pool, as any tensor made here would.";

PyObject* launch_py(PyObject*, PyObject* const* a, Py_ssize_t n, PyObject* names) {
    HANDLE_TH_ERRORS
    Kwargs kw;
    PyObject* in[4];
    if (!kw.parse(names, a + n) || !kw.operands(a, n, "flash_attn_ext", in)) return nullptr;
    const at::Tensor* q = tensor_of(in[0], "q");
    if (!q) return nullptr;
    if (!q->is_cuda()) {
        PyErr_SetString(PyExc_ValueError, "flash_attn_ext takes CUDA tensors; use flash_attn_ext_host for host buffers");
        return nullptr;
    }
    const c10::cuda::CUDAGuard guard(q->device());
    PyObject* out = kw.v[kOut];
    at::Tensor made;
    if (!out) {
        if (q->dim() != 4) {
            PyErr_SetString(PyExc_ValueError, "q is (B, H, Tq, hd)");
            return nullptr;
        }
        made = at::detail::empty_cuda({q->size(0), q->size(2), q->size(1), q->size(3)}, at::kFloat, q->device(), std::nullopt);
    }
    const at::Tensor* dst = out ? tensor_of(out, "out") : &made;
    Operands op;
    if (!dst || !op.fill(in[0], in[1], in[2], in[3], kw) || !describe(*dst, -1, &op.dst)) return nullptr;
    Scratch ws{at::Tensor(), q->device(), nullptr, 0, nullptr, nullptr};
    if (kw.v[kWorkspace]) {
        const at::Tensor* w = tensor_of(kw.v[kWorkspace], "workspace");
        if (!w) return nullptr;
        ws.given = w->data_ptr(), ws.given_bytes = (size_t)w->numel();
    }
    void* st = nullptr;
    if (!kw.v[kStream]) st = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
    else if (!stream_of(kw.v[kStream], &st)) return nullptr;
    ws.stream = st;
    int rc;
    Py_BEGIN_ALLOW_THREADS   // a full launch queue blocks: other host threads go on meanwhile
    rc = b200_fattn_launch_alloc(&op.q, &op.k, &op.v, op.mask_p(), &op.dst, &op.params, &op.ext, scratch_alloc, &ws, st);
    Py_END_ALLOW_THREADS
    if (ws.error) std::rethrow_exception(ws.error);   // torch.OutOfMemoryError, as from any other allocation
    if (rc) return raise_code(rc, "b200_fattn_launch");
    if (!out) return THPVariable_Wrap(std::move(made));
    Py_INCREF(out);
    return out;
    END_HANDLE_TH_ERRORS
}

const char kHostDoc[] =
    "flash_attn_ext_host(q, k, v, mask=None, *, out=None, **kw)\n--\n\n"
    "Host (CPU, ideally pinned) tensors in, host tensor out: H2D, compute, D2H inside one C call.";

PyObject* forward_host_py(PyObject*, PyObject* const* a, Py_ssize_t n, PyObject* names) {
    HANDLE_TH_ERRORS
    Kwargs kw;
    PyObject* in[4];
    if (!kw.parse(names, a + n) || !kw.operands(a, n, "flash_attn_ext_host", in)) return nullptr;
    const at::Tensor* q = tensor_of(in[0], "q");
    if (!q) return nullptr;
    PyObject* out = kw.v[kOut];
    at::Tensor made;
    if (!out) {
        if (q->dim() != 4) {
            PyErr_SetString(PyExc_ValueError, "q is (B, H, Tq, hd)");
            return nullptr;
        }
        made = at::empty({q->size(0), q->size(2), q->size(1), q->size(3)}, q->options().dtype(at::kFloat));
    }
    const at::Tensor* dst = out ? tensor_of(out, "out") : &made;
    Operands op;
    if (!dst || !op.fill(in[0], in[1], in[2], in[3], kw) || !describe(*dst, -1, &op.dst)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_fattn_forward_host(&op.q, &op.k, &op.v, op.mask_p(), &op.dst, &op.params, &op.ext);
    Py_END_ALLOW_THREADS
    if (rc) return raise_code(rc, "b200_fattn_forward_host");
    if (!out) return THPVariable_Wrap(std::move(made));
    Py_INCREF(out);
    return out;
    END_HANDLE_TH_ERRORS
}

// (cache address, layer, k_new, v_new, pos, pos0, stream)
PyObject* kv_append_py(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 7) {
        PyErr_SetString(PyExc_TypeError, "kv_append takes 7 arguments");
        return nullptr;
    }
    HANDLE_TH_ERRORS
    b200_kv_cache* kv = (b200_kv_cache*)PyLong_AsVoidPtr(a[0]);
    const long layer = PyLong_AsLong(a[1]);
    if (PyErr_Occurred()) return nullptr;
    PyObject* p0 = PyNumber_Long(a[5]);   // int(pos0): floats as well
    if (!p0) return nullptr;
    const long pos0 = PyLong_AsLong(p0);
    Py_DECREF(p0);
    if (PyErr_Occurred()) return nullptr;
    const at::Tensor *k = tensor_of(a[2], "k_new"), *v = k ? tensor_of(a[3], "v_new") : nullptr;
    b200_tensor tk, tv;
    if (!v || !describe(*k, -1, &tk) || !describe(*v, -1, &tv)) return nullptr;
    const int32_t* pos = nullptr;
    if (a[4] != Py_None && !PyObject_HasAttrString(a[4], "data_ptr")) {   // (read by the kernel: a numpy array has no device address)
        PyErr_Format(PyExc_TypeError, "pos is a torch tensor, not %s", Py_TYPE(a[4])->tp_name);
        return nullptr;
    }
    if (a[4] != Py_None && !address_of(a[4], &pos)) return nullptr;
    if (a[6] == Py_None && !k->is_cuda()) {
        PyErr_SetString(PyExc_ValueError, "kv_append takes CUDA tensors");
        return nullptr;
    }
    void* st = nullptr;
    if (a[6] == Py_None) st = c10::cuda::getCurrentCUDAStream(k->device().index()).stream();
    else if (!stream_of(a[6], &st)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = b200_kv_append(kv, (int)layer, &tk, &tv, pos, (int32_t)pos0, st);
    Py_END_ALLOW_THREADS
    if (rc) return raise_code(rc, "b200_kv_append");
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"flash_attn_ext", (PyCFunction)(void (*)(void))launch_py, METH_FASTCALL | METH_KEYWORDS, kLaunchDoc},
    {"flash_attn_ext_host", (PyCFunction)(void (*)(void))forward_host_py, METH_FASTCALL | METH_KEYWORDS, kHostDoc},
    {"kv_append", (PyCFunction)(void (*)(void))kv_append_py, METH_FASTCALL, "rows of a KV cache"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_op", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_op(void) {
    for (int i = 0; i < kKeys; i++)
        if (!(g_keys[i] = PyUnicode_InternFromString(kKeyNames[i]))) return nullptr;
    return PyModule_Create(&kModule);
}
