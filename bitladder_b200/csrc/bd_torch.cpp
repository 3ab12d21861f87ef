// The operators' calls on torch tensors, from the Python arguments to the C entry points without interpreted code in
// between: bit_decode_interface.py hands a call over, and gets None back for every call that is not plainly valid (a
// wrong shape, a tensor subclass, an argument of another type, a workspace that has to be grown).  Such a call is
// checked, refused or served by the Python code, so this file raises nothing and decides nothing about errors; the two
// have to accept the same calls and fill the same argument blocks.
//
// Why: the checks and the argument block cost 20 to 30 us of interpreter per call, more than the kernels of a small step
// (a fwd_kvcache_int call of 1 x 4096 tokens, 32/32 heads: 34.9 us a pass before, 13.0 with this file;
// kvcache_pack_int of one block of 8 sequences 27.5 -> 6.4 us).
//
// Nothing is kept between calls; the workspaces live in the dictionary that the Python code owns.  The interpreter lock is
// let go around allocations and launches (a launch waits where the stream's queue is full, and what it waits for may be a
// host function that needs the lock), as ctypes does: what is used there is owned by this call, not borrowed.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/bitdecode.h"

namespace {

// Entry points of the library that the Python package has loaded.
int (*g_decode)(const bd_decode_args *, bd_stream_t) = nullptr;
int (*g_pack)(const bd_pack_args *, bd_stream_t) = nullptr;
size_t (*g_workspace_bytes)(const bd_decode_args *) = nullptr;

struct NotPlain {};      // the Python code takes the call
inline void need(bool ok) {
    if (!ok) throw NotPlain();
}

// Other Python threads run while one of these lives; nothing of the interpreter may be touched.
struct Unlocked {
    PyThreadState *state = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked &) = delete;
    ~Unlocked() { PyEval_RestoreThread(state); }
};

// A plain CUDA tensor on `dev` (an index below 0: any, which it then becomes).
const at::Tensor &tensor(PyObject *o, c10::DeviceIndex &dev) {
    need(THPVariable_CheckExact(o));
    const at::Tensor &t = THPVariable_Unpack(o);
    need(t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.has_storage());
    if (dev < 0) dev = t.get_device();
    need(t.get_device() == dev);
    return t;
}
const at::Tensor *optional_tensor(PyObject *o, c10::DeviceIndex &dev) { return o == Py_None ? nullptr : &tensor(o, dev); }

int64_t integer(PyObject *o) {
    need(PyLong_CheckExact(o));
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); throw NotPlain(); }
    return v;
}
bool boolean(PyObject *o) {
    need(PyBool_Check(o));
    return o == Py_True;
}

void config(PyObject *mode, PyObject *group, PyObject *bits, int &g, int &nbits) {
    need(PyUnicode_CheckExact(mode) && PyUnicode_CompareWithASCIIString(mode, "k-channel") == 0);
    const int64_t gg = integer(group), bb = integer(bits);
    need((bb == 2 || bb == 4) && (gg == 32 || gg == 64 || gg == 128));
    g = int(gg);
    nbits = int(bb);
}

int dtype_code(at::ScalarType t) {
    if (t == at::kHalf) return BD_FP16;
    if (t == at::kBFloat16) return BD_BF16;
    need(t == at::kFloat);
    return BD_FP32;
}
bool half_type(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }

// Dims 1.. laid out densely (dim 0 may have any stride).
bool rows_contiguous(const at::Tensor &t) {
    int64_t expected = 1;
    for (int64_t i = t.dim() - 1; i >= 1; --i) {
        if (t.size(i) != 1 && t.stride(i) != expected) return false;
        expected *= t.size(i);
    }
    return true;
}
bool has_shape(const at::Tensor &t, int64_t a, int64_t b, int64_t c, int64_t d) {
    return t.dim() == 4 && t.size(0) == a && t.size(1) == b && t.size(2) == c && t.size(3) == d;
}

struct Packed {
    int64_t b, s_cap, h_k;
};
Packed packed(const at::Tensor &kp, const at::Tensor &kprm, const at::Tensor &vp, const at::Tensor &vprm, int bits, int group) {
    const int64_t pn = 16 / bits, nb = 32 * pn;
    for (const at::Tensor *t : {&kp, &vp}) need(t->scalar_type() == at::kUInt16 || t->scalar_type() == at::kShort);
    for (const at::Tensor *t : {&kprm, &vprm}) need(t->scalar_type() == at::kFloat);
    need(vp.dim() == 4);
    const Packed r{vp.size(0), vp.size(1), vp.size(2)};
    need(vp.size(3) * pn == 128 && r.s_cap % nb == 0);
    need(has_shape(kp, r.b, r.s_cap / pn, r.h_k, 128) && has_shape(kprm, r.b, r.s_cap / group, r.h_k, 128) &&
         has_shape(vprm, r.b, 128 / group, r.h_k, r.s_cap));
    need(rows_contiguous(kp) && rows_contiguous(kprm) && rows_contiguous(vp) && rows_contiguous(vprm));
    return r;
}

const int32_t *lengths(const at::Tensor &t, int64_t b) {
    need(t.scalar_type() == at::kInt && t.numel() == b && t.is_contiguous());
    return static_cast<const int32_t *>(t.data_ptr());
}

// The dictionary's workspace for this device and stream, if it is there, large enough and cleared for this layout.  The
// caller owns it: another thread may put a larger one in its place while this call runs.
at::Tensor workspace(PyObject *dict, c10::DeviceIndex dev, void *stream, bd_decode_args &a) {
    const size_t bytes = g_workspace_bytes(&a);
    need(bytes > 0 && PyDict_CheckExact(dict));
    PyObject *key = Py_BuildValue("(iK)", int(dev), (unsigned long long)(uintptr_t)stream);
    if (!key) { PyErr_Clear(); throw NotPlain(); }
    PyObject *entry = PyDict_GetItemWithError(dict, key);            // borrowed
    Py_DECREF(key);
    if (!entry) { PyErr_Clear(); throw NotPlain(); }
    need(PyList_CheckExact(entry) && PyList_GET_SIZE(entry) == 2);
    PyObject *layout = PyList_GET_ITEM(entry, 1);
    need(PyTuple_CheckExact(layout) && PyTuple_GET_SIZE(layout) == 3);
    need(integer(PyTuple_GET_ITEM(layout, 0)) == a.b && integer(PyTuple_GET_ITEM(layout, 1)) == a.h_k &&
         boolean(PyTuple_GET_ITEM(layout, 2)) == (a.cache_seqlens != nullptr));
    const at::Tensor &ws = tensor(PyList_GET_ITEM(entry, 0), dev);
    need(size_t(ws.numel()) >= bytes);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = size_t(ws.numel());
    return ws;
}

PyObject *decode_call(PyObject *const *o) {
    c10::DeviceIndex dev = -1;
    const at::Tensor &q = tensor(o[1], dev), &kp = tensor(o[2], dev), &kprm = tensor(o[3], dev), &vp = tensor(o[4], dev),
                     &vprm = tensor(o[5], dev);
    const at::Tensor *table = optional_tensor(o[6], dev);
    need(PyFloat_CheckExact(o[7]) || PyLong_CheckExact(o[7]));
    const double scale = PyFloat_AsDouble(o[7]);
    if (scale == -1.0 && PyErr_Occurred()) { PyErr_Clear(); throw NotPlain(); }
    int group, bits;
    config(o[8], o[9], o[10], group, bits);
    const at::Tensor *k_res = optional_tensor(o[11], dev), *v_res = optional_tensor(o[12], dev), *res_lens = optional_tensor(o[13], dev),
                     *cache_seqlens = optional_tensor(o[14], dev);
    const bool return_lse = boolean(o[16]);
    need(o[17] == Py_None || THPDtype_Check(o[17]));
    const at::Tensor *k_new = optional_tensor(o[19], dev), *v_new = optional_tensor(o[20], dev);
    const bool advance = boolean(o[21]);
    const at::Tensor *cos = optional_tensor(o[22], dev), *sin = optional_tensor(o[23], dev);

    const at::ScalarType type = q.scalar_type();
    need(half_type(type) && q.dim() == 4 && q.size(1) == 1 && q.size(3) == 128 && q.stride(3) == 1);
    const Packed pk = packed(kp, kprm, vp, vprm, bits, group);
    bd_decode_args a = {};
    int64_t b = pk.b, s_max = pk.s_cap;
    if (table) {
        need(table->scalar_type() == at::kInt && table->dim() == 2 && table->stride(1) == 1 && pk.s_cap % 256 == 0);
        b = table->size(0);
        s_max = pk.s_cap * table->size(1);
        a.block_table = static_cast<const int32_t *>(table->data_ptr());
        a.block_table_stride = int32_t(table->stride(0));
        a.num_pages = int32_t(pk.b);
    }
    const int64_t h = q.size(2), h_k = pk.h_k;
    need(q.size(0) == b && b > 0 && h_k > 0 && h > 0 && h % h_k == 0 && h / h_k <= 16);
    const int64_t s = o[15] == Py_None ? s_max : integer(o[15]);
    need(s >= 0 && s <= s_max && s_max <= INT32_MAX && b <= INT32_MAX && h <= INT32_MAX);
    a.q = q.data_ptr();
    a.q_stride_b = q.stride(0); a.q_stride_h = q.stride(2);
    a.k_pack = kp.data_ptr(); a.k_params = kprm.data_ptr(); a.v_pack = vp.data_ptr(); a.v_params = vprm.data_ptr();
    a.k_pack_stride_b = kp.stride(0); a.k_params_stride_b = kprm.stride(0); a.v_pack_stride_b = vp.stride(0);
    a.v_params_stride_b = vprm.stride(0); a.v_params_stride_g = vprm.stride(1); a.v_params_stride_h = vprm.stride(2);
    if (cache_seqlens) a.cache_seqlens = lengths(*cache_seqlens, b);
    need((k_res != nullptr) == (v_res != nullptr) && (k_new != nullptr) == (v_new != nullptr) && (cos != nullptr) == (sin != nullptr));
    if (k_res) {
        need(k_res->scalar_type() == type && v_res->scalar_type() == type && k_res->dim() == 4 && v_res->sizes() == k_res->sizes() &&
             v_res->strides() == k_res->strides());
        need(k_res->size(0) == b && k_res->size(1) <= 256 && k_res->size(2) == h_k && k_res->size(3) == 128 && k_res->stride(3) == 1);
        a.k_res = k_res->data_ptr(); a.v_res = v_res->data_ptr();
        a.res_stride_b = k_res->stride(0); a.res_stride_s = k_res->stride(1); a.res_stride_h = k_res->stride(2);
        a.res_len = int32_t(k_res->size(1));
        if (res_lens) a.res_lens = lengths(*res_lens, b);
    }
    if (k_new) {
        need(k_res && res_lens && k_new->scalar_type() == type && v_new->scalar_type() == type && has_shape(*k_new, b, 1, h_k, 128) &&
             v_new->sizes() == k_new->sizes() && v_new->strides() == k_new->strides() && k_new->stride(3) == 1);
        a.k_new = k_new->data_ptr(); a.v_new = v_new->data_ptr();
        a.new_stride_b = k_new->stride(0); a.new_stride_h = k_new->stride(2);
    }
    a.b = int32_t(b); a.h = int32_t(h); a.h_k = int32_t(h_k); a.d = 128;
    a.s = int32_t(s); a.s_cap = int32_t(pk.s_cap);
    a.bits = bits; a.group = group;
    a.dtype = dtype_code(type);
    const at::ScalarType out_type = o[17] == Py_None ? type : reinterpret_cast<THPDtype *>(o[17])->scalar_type;
    a.out_dtype = dtype_code(out_type);
    a.softmax_scale = float(scale);
    const int64_t splits = integer(o[18]);
    need(splits >= INT32_MIN && splits <= INT32_MAX);
    a.num_splits = int32_t(splits);
    if (advance) {
        need(k_new && cache_seqlens && res_lens && !table && k_res->size(1) >= 32 * (16 / bits));
        a.advance = 1;
    }
    if (cos) {
        need(k_new && cos->scalar_type() == type && sin->scalar_type() == type && cos->dim() == 2 && cos->sizes() == sin->sizes() &&
             cos->is_contiguous() && sin->is_contiguous());
        const int64_t dim = 2 * cos->size(1);
        need(dim > 0 && dim <= 128 && dim % 16 == 0 && cos->size(0) <= INT32_MAX);
        a.rotary_cos = cos->data_ptr(); a.rotary_sin = sin->data_ptr();
        a.rotary_dim = int32_t(dim);
        a.rotary_interleaved = boolean(o[24]) ? 1 : 0;
        a.rotary_positions = int32_t(cos->size(0));
    }

    c10::cuda::CUDAGuard guard(dev);
    void *stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    const at::Tensor ws = workspace(o[0], dev, stream, a);
    const at::TensorOptions options = q.options();
    at::Tensor out, lse;
    {
        Unlocked unlocked;
        out = at::empty({b, 1, h, 128}, options.dtype(out_type));
        a.out = out.data_ptr();
        a.out_stride_b = out.stride(0); a.out_stride_h = out.stride(2);
        if (return_lse) {
            lse = at::empty({b, h}, options.dtype(at::kFloat));
            a.lse = static_cast<float *>(lse.data_ptr());
        }
        need(g_decode(&a, stream) == BD_OK);
    }
    if (!return_lse) return THPVariable_Wrap(std::move(out));
    PyObject *po = THPVariable_Wrap(std::move(out)), *pl = THPVariable_Wrap(std::move(lse));
    PyObject *pair = PyTuple_New(2);
    PyTuple_SET_ITEM(pair, 0, po);
    PyTuple_SET_ITEM(pair, 1, pl);
    return pair;
}

PyObject *pack_call(PyObject *const *o) {
    c10::DeviceIndex dev = -1;
    const at::Tensor &k = tensor(o[0], dev), &kp = tensor(o[1], dev), &kprm = tensor(o[2], dev), &v = tensor(o[3], dev),
                     &vp = tensor(o[4], dev), &vprm = tensor(o[5], dev);
    int group, bits;
    config(o[6], o[7], o[8], group, bits);
    const int64_t offset = integer(o[9]);
    const bool approx = boolean(o[10]);
    const at::ScalarType type = k.scalar_type();
    need(half_type(type) && v.scalar_type() == type && k.dim() == 4 && k.sizes() == v.sizes() && k.stride(3) == 1 && v.stride(3) == 1);
    const Packed pk = packed(kp, kprm, vp, vprm, bits, group);
    const int64_t nb = 32 * (16 / bits), s = k.size(1);
    need(k.size(0) == pk.b && k.size(2) == pk.h_k && k.size(3) == 128);
    need(s > 0 && s % nb == 0 && offset >= 0 && offset % nb == 0 && offset + s <= pk.s_cap && pk.s_cap <= INT32_MAX && pk.b <= INT32_MAX);
    bd_pack_args a = {};
    a.k = k.data_ptr(); a.v = v.data_ptr();
    a.k_stride_b = k.stride(0); a.k_stride_s = k.stride(1); a.k_stride_h = k.stride(2);
    a.v_stride_b = v.stride(0); a.v_stride_s = v.stride(1); a.v_stride_h = v.stride(2);
    a.k_pack = kp.data_ptr(); a.k_params = kprm.data_ptr(); a.v_pack = vp.data_ptr(); a.v_params = vprm.data_ptr();
    a.k_pack_stride_b = kp.stride(0); a.k_params_stride_b = kprm.stride(0); a.v_pack_stride_b = vp.stride(0);
    a.v_params_stride_b = vprm.stride(0); a.v_params_stride_g = vprm.stride(1); a.v_params_stride_h = vprm.stride(2);
    a.b = int32_t(pk.b); a.s = int32_t(s); a.h_k = int32_t(pk.h_k); a.d = 128;
    a.dst_token_offset = int32_t(offset);
    a.bits = bits; a.group = group; a.dtype = dtype_code(type);
    a.flags = approx ? BD_PACK_APPROX_DIV : 0;
    c10::cuda::CUDAGuard guard(dev);
    {
        Unlocked unlocked;
        need(g_pack(&a, c10::cuda::getCurrentCUDAStream(dev).stream()) == BD_OK);
    }
    Py_RETURN_TRUE;
}

// Nothing gets out as an exception: what did not go through is the Python code's call.
template <PyObject *(*F)(PyObject *const *), Py_ssize_t N>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    if (n == N && g_decode) {
        try {
            return F(args);
        } catch (...) {
        }
    }
    Py_RETURN_NONE;
}

// bind(decode, pack, workspace_bytes): addresses of the loaded library's entry points.
PyObject *bind(PyObject *, PyObject *args) {
    unsigned long long d, p, w;
    if (!PyArg_ParseTuple(args, "KKK", &d, &p, &w)) return nullptr;
    g_pack = reinterpret_cast<decltype(g_pack)>(uintptr_t(p));
    g_workspace_bytes = reinterpret_cast<decltype(g_workspace_bytes)>(uintptr_t(w));
    g_decode = reinterpret_cast<decltype(g_decode)>(uintptr_t(d));
    Py_RETURN_NONE;
}

// step(args address, device index): bd_decode with a prepared argument block on the device's current stream.
PyObject *step(PyObject *, PyObject *const *args, Py_ssize_t n) {
    if (n != 2) {
        PyErr_SetString(PyExc_TypeError, "step(args, device)");
        return nullptr;
    }
    const void *a = PyLong_AsVoidPtr(args[0]);
    const long dev = PyLong_AsLong(args[1]);
    if (PyErr_Occurred()) return nullptr;
    int rc = BD_ERR_CUDA;
    try {
        Unlocked unlocked;
        c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(dev));
        rc = g_decode(static_cast<const bd_decode_args *>(a), c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream());
    } catch (...) {
    }
    return PyLong_FromLong(rc);
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<decode_call, 25>)), METH_FASTCALL, nullptr},
    {"pack", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<pack_call, 11>)), METH_FASTCALL, nullptr},
    {"step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&step)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// BUILT_FOR: the torch and the interpreter whose headers were compiled in; bit_decode_interface.py takes no other.
PyMODINIT_FUNC PyInit__torch_calls(void) {
    PyObject *m = PyModule_Create(&kModule);
    if (m && PyModule_AddStringConstant(m, "BUILT_FOR", BD_BUILT_FOR) < 0) Py_CLEAR(m);
    return m;
}
