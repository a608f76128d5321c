// Host path of the package's tensor-level calls: a CPython module that takes torch tensors,
// checks and converts them, allocates outputs and calls the C ABI (include/ftq_b200.h) on the
// caller's current stream.
//
// Why it exists: a decode step of a small batch is two calls whose kernels run for 10-20 us, and
// the same argument handling written in Python over ctypes kept the host busy for 70 us (store +
// decode of one sequence; 28 us for a store alone, 60 us for a quantizer round trip) -- the GPU
// idled for most of the step.  Here a call costs 3-5 us on top of its kernel launches.
//
// The module holds no state of its own besides the C ABI's addresses (bind()) and host copies of
// small tables that the caller passes as tensors (dropped with the tensor).
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/ftq_b200.h"

namespace {

// ------------------------------------------------------------------ the C ABI, bound at import
#define FTQ_BOUND(X)                                                                       \
    X(ftq_encode) X(ftq_decode_dense) X(ftq_rht) X(ftq_decode_workspace_bytes)             \
    X(ftq_flash_decode) X(ftq_paged_store) X(ftq_paged_decode_attn) X(ftq_tq_store_layers) \
    X(ftq_tq_decode_layers_ws) X(ftq_tq_decode_layers_workspace_bytes) X(ftq_paged_chunk_workspace_bytes) X(ftq_paged_chunk_attn)
struct Api {
#define X(name) decltype(&::name) name = nullptr;
    FTQ_BOUND(X)
#undef X
} api;
PyObject* g_check = nullptr;        // _lib.check(rc, name): raises what the status stands for
PyObject* g_get_workspace = nullptr;  // kernels.get_workspace(device, nbytes)
PyObject* g_workspaces = nullptr;     // kernels._workspaces
PyObject* g_host_table = nullptr;     // kernels._host_table: fp32 copy of an array of any type and strides

struct PyError {};  // a Python exception is set

struct NoGil {
    PyThreadState* s = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(s); }
};

[[noreturn]] void raise(PyObject* type, const std::string& msg) {
    PyErr_SetString(type, msg.c_str());
    throw PyError{};
}

void check(int rc, const char* what) {
    if (rc == FTQ_OK) return;
    PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
    if (!r) throw PyError{};
    Py_DECREF(r);
    raise(PyExc_RuntimeError, std::string(what) + " failed");
}

const at::Tensor& tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, std::string(name) + " must be a tensor");
    return THPVariable_Unpack(o);
}
const at::Tensor& cuda_tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o) || !THPVariable_Unpack(o).is_cuda())
        raise(PyExc_RuntimeError, std::string(name) +
              " must be a CUDA tensor: fused_turboquant_b200 has no CPU path "
              "(build libftq_b200.so and run on a B200)");
    return THPVariable_Unpack(o);
}
int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return FTQ_F32;
        case at::kHalf: return FTQ_F16;
        case at::kBFloat16: return FTQ_BF16;
        default: return -1;
    }
}
int out_dtype_code(const at::Tensor& t) {
    const int c = dtype_code(t.scalar_type());
    if (c < 0) raise(PyExc_KeyError, c10::toString(t.scalar_type()));
    return c;
}
// fp32 / fp16 / bf16 as they are, anything else as fp32
at::Tensor supported(const at::Tensor& t) {
    return dtype_code(t.scalar_type()) < 0 ? t.to(at::kFloat) : t;
}
at::Tensor as_i32(PyObject* o, const char* name, const at::Device& dev) {
    const at::Tensor& t = tensor(o, name);
    if (t.scalar_type() == at::kInt && t.device() == dev && t.is_contiguous()) return t;
    return t.to(dev, at::kInt).contiguous();
}
at::Tensor as_i64(PyObject* o, const char* name, const at::Device& dev) {
    const at::Tensor& t = tensor(o, name);
    if (t.scalar_type() == at::kLong && t.device() == dev && t.is_contiguous()) return t;
    return t.to(dev, at::kLong).contiguous();
}
long long as_int(PyObject* o) {
    long long v;
    if (PyLong_Check(o)) {
        v = PyLong_AsLongLong(o);
    } else {   // anything with __int__ (numpy scalars, one-element tensors)
        PyObject* i = PyNumber_Long(o);
        if (!i) throw PyError{};
        v = PyLong_AsLongLong(i);
        Py_DECREF(i);
    }
    if (v == -1 && PyErr_Occurred()) throw PyError{};
    return v;
}
double as_double(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyError{};
    return v;
}
bool as_bool(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PyError{};
    return v != 0;
}
template <class T = uint8_t>
const T* ptr(const at::Tensor& t) { return static_cast<const T*>(t.const_data_ptr()); }
template <class T = uint8_t>
T* mptr(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }
void* stream_of(const at::Device& d) {
    return c10::cuda::getCurrentCUDAStream(d.index()).stream();
}
at::Tensor empty(at::IntArrayRef size, at::ScalarType t, const at::Device& d) {
    return at::empty(size, at::TensorOptions().dtype(t).device(d));
}

// ------------------------------------------------------------------ small host tables
// Contiguous fp32 arrays are read in place, other arrays converted; a tensor's values are copied to
// the host once and kept while the tensor is alive and unmodified (as kernels._host_table does for the
// other callers).
struct CachedTable {
    c10::weak_intrusive_ptr<c10::TensorImpl> owner;
    uint32_t version;
    std::vector<float> values;
};
std::mutex table_mu;
std::unordered_map<const void*, CachedTable>* tables = new std::unordered_map<const void*, CachedTable>;

struct Table {
    const float* p = nullptr;
    Py_buffer view{};
    std::vector<float> own;
    explicit Table(PyObject* o) {
        if (o == nullptr || o == Py_None) return;
        if (THPVariable_Check(o)) { from_tensor(THPVariable_Unpack(o)); return; }
        if (from_buffer(o)) return;
        PyObject* c = PyObject_CallOneArg(g_host_table, o);
        if (!c) throw PyError{};
        const bool ok = from_buffer(c);   // (the view holds the array)
        Py_DECREF(c);
        if (!ok) raise(PyExc_TypeError, "a table must be an array or a tensor of numbers");
    }
    Table(const Table&) = delete;
    ~Table() { if (view.obj) PyBuffer_Release(&view); }

   private:
    bool from_buffer(PyObject* o) {
        if (PyObject_GetBuffer(o, &view, PyBUF_CONTIG_RO | PyBUF_FORMAT) != 0) {
            PyErr_Clear();
            return false;
        }
        if (view.itemsize == 4 && view.format && view.format[0] == 'f') {
            p = static_cast<const float*>(view.buf);
            return true;
        }
        PyBuffer_Release(&view);
        view.obj = nullptr;
        return false;
    }
    void from_tensor(const at::Tensor& t) {
        const bool keep = !t.is_inference();
        const void* key = t.unsafeGetTensorImpl();
        if (keep) {
            std::lock_guard<std::mutex> lock(table_mu);
            auto it = tables->find(key);
            if (it != tables->end()) {
                if (!it->second.owner.expired() && it->second.version == t._version()) {
                    own = it->second.values;   // (at most 256 floats)
                    p = own.data();
                    return;
                }
                tables->erase(it);
            }
        }
        at::Tensor h;
        {
            NoGil nogil;   // may wait for the device
            h = t.detach().to(at::kCPU, at::kFloat).contiguous();
        }
        own.assign(h.const_data_ptr<float>(), h.const_data_ptr<float>() + h.numel());
        p = own.data();
        if (keep) {
            std::lock_guard<std::mutex> lock(table_mu);
            for (auto it = tables->begin(); it != tables->end();)
                it = it->second.owner.expired() ? tables->erase(it) : std::next(it);
            tables->insert_or_assign(key, CachedTable{
                c10::weak_intrusive_ptr<c10::TensorImpl>(t.getIntrusivePtr()),
                static_cast<uint32_t>(t._version()), own});
        }
    }
};

// Scratch of the current (device, stream), shared with the Python callers (kernels.get_workspace).
at::Tensor workspace(PyObject* given, const at::Device& dev, void* stream, size_t need) {
    if (given != Py_None) return tensor(given, "workspace");
    PyObject* key = Py_BuildValue("(iK)", static_cast<int>(dev.index()),
                                  static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)));
    if (!key) throw PyError{};
    PyObject* hit = PyDict_GetItemWithError(g_workspaces, key);
    Py_DECREF(key);
    if (hit && THPVariable_Check(hit) &&
        static_cast<size_t>(THPVariable_Unpack(hit).numel()) >= need)
        return THPVariable_Unpack(hit);
    if (PyErr_Occurred()) throw PyError{};
    PyObject* d = THPDevice_New(dev);
    PyObject* r = PyObject_CallFunction(g_get_workspace, "OK", d, static_cast<unsigned long long>(need));
    Py_DECREF(d);
    if (!r) throw PyError{};
    at::Tensor t = THPVariable_Unpack(r);
    Py_DECREF(r);
    return t;
}

// ------------------------------------------------------------------ attributes of a PagedKVPool
struct Ref {
    PyObject* o;
    explicit Ref(PyObject* x) : o(x) { if (!o) throw PyError{}; }
    Ref(const Ref&) = delete;
    ~Ref() { Py_DECREF(o); }
};
#define FTQ_NAMES(X)                                                                              \
    X(pool) X(num_blocks) X(num_kv_heads) X(head_dim) X(key_bits) X(value_bits) X(page_bytes)     \
    X(signs) X(bounds_k) X(bounds_v) X(levels_k) X(levels_v) X(_last_decode)
struct Names {
#define X(name) PyObject* name = nullptr;
    FTQ_NAMES(X)
#undef X
} names;
long long int_attr(PyObject* self, PyObject* name) {
    Ref r(PyObject_GetAttr(self, name));
    return as_int(r.o);
}

struct Pool {
    at::Tensor pool;
    int64_t num_blocks, hkv, d, kb, vb, layer_stride, n_layers;
    explicit Pool(PyObject* self) {
        Ref p(PyObject_GetAttr(self, names.pool));
        pool = tensor(p.o, "pool");
        num_blocks = int_attr(self, names.num_blocks);
        hkv = int_attr(self, names.num_kv_heads);
        d = int_attr(self, names.head_dim);
        kb = int_attr(self, names.key_bits);
        vb = int_attr(self, names.value_bits);
        layer_stride = num_blocks * hkv * int_attr(self, names.page_bytes);
        n_layers = pool.size(0);
    }
    uint8_t* base(PyObject* layer) const {
        uint8_t* p = mptr(pool);
        if (layer == Py_None) return p;
        long long l = as_int(layer);
        if (l < -n_layers || l >= n_layers)
            raise(PyExc_IndexError, "layer " + std::to_string(l) + " is out of range");
        return p + (l < 0 ? l + n_layers : l) * pool.stride(0);
    }
};

void want_args(Py_ssize_t n, Py_ssize_t want, const char* what) {
    if (n != want) raise(PyExc_TypeError, std::string(what) + ": wrong number of arguments");
}

// paged_store(self, key, value, slot_mapping, layer)
PyObject* paged_store(PyObject* const* a) {
    PyObject* self = a[0];
    at::Tensor key = cuda_tensor(a[1], "key"), value = tensor(a[2], "value");
    if (dtype_code(key.scalar_type()) < 0) { key = key.to(at::kFloat); value = value.to(at::kFloat); }
    if (!key.is_contiguous()) key = key.contiguous();
    if (!value.is_contiguous()) value = value.contiguous();
    if (value.scalar_type() != key.scalar_type()) value = value.to(key.scalar_type());
    const at::Device dev = key.device();
    const at::Tensor sm = as_i64(a[3], "slot_mapping", dev);
    const Pool p(self);
    const bool all = a[4] == Py_None;
    if (key.dim() < (all ? 2 : 1)) raise(PyExc_IndexError, "key has too few dimensions");
    const int64_t L = all ? key.size(0) : 1, n = key.size(all ? 1 : 0);
    uint8_t* base = p.base(a[4]);
    Ref so(PyObject_GetAttr(self, names.signs)), ko(PyObject_GetAttr(self, names.bounds_k)),
        vo(PyObject_GetAttr(self, names.bounds_v));
    const Table signs(so.o), bk(ko.o), bv(vo.o);
    const c10::cuda::CUDAGuard guard(dev);
    void* st = stream_of(dev);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_paged_store(ptr<void>(key), ptr<void>(value), dtype_code(key.scalar_type()), n,
                                 p.hkv, p.d, p.hkv * p.d, p.d, p.kb, p.vb, signs.p, bk.p, bv.p, base,
                                 p.num_blocks, ptr<int64_t>(sm), L, n * p.hkv * p.d, p.layer_stride, st);
    }
    check(rc, "ftq_paged_store");
    Py_RETURN_NONE;
}

// paged_decode(self, q, block_table, seq_lens, max_seq_len, scale, layer, out, workspace)
PyObject* paged_decode(PyObject* const* a) {
    PyObject* self = a[0];
    at::Tensor q = supported(cuda_tensor(a[1], "q"));
    if (!q.is_contiguous()) q = q.contiguous();
    const Pool p(self);
    const bool all = a[6] == Py_None;
    if (q.dim() != (all ? 4 : 3))
        raise(PyExc_ValueError, all ? "q must be [n_layers, B, Hq, D]" : "q must be [B, Hq, D]");
    const int64_t L = all ? q.size(0) : 1, B = q.size(-3), Hq = q.size(-2), D = q.size(-1);
    const double scale = a[5] == Py_None ? std::pow(static_cast<double>(D), -0.5) : as_double(a[5]);
    const at::Device dev = q.device();
    const at::Tensor bt = as_i32(a[2], "block_table", dev), sl = as_i32(a[3], "seq_lens", dev);
    const long long max_seq = as_int(a[4]);
    if (bt.dim() < 2) raise(PyExc_IndexError, "block_table must be [B, max_blocks]");
    const c10::cuda::CUDAGuard guard(dev);
    const at::Tensor out = a[7] == Py_None ? empty(q.sizes(), q.scalar_type(), dev) : tensor(a[7], "out");
    const int oc = out_dtype_code(out);
    void* st = stream_of(dev);
    const at::Tensor ws = workspace(a[8], dev, st,
                                    api.ftq_decode_workspace_bytes(B, Hq, p.hkv, p.d, max_seq, L));
    uint8_t* base = p.base(a[6]);
    Ref so(PyObject_GetAttr(self, names.signs)), ko(PyObject_GetAttr(self, names.levels_k)),
        vo(PyObject_GetAttr(self, names.levels_v));
    const Table signs(so.o), lk(ko.o), lv(vo.o);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_paged_decode_attn(
            ptr<void>(q), dtype_code(q.scalar_type()), mptr<void>(out), oc, base, p.num_blocks,
            p.layer_stride, L, ptr<int32_t>(bt), bt.size(1), ptr<int32_t>(sl), max_seq, B, Hq, p.hkv,
            D, p.kb, p.vb, lk.p, lv.p, signs.p, static_cast<float>(scale), mptr<void>(ws), ws.numel(), st);
    }
    check(rc, "ftq_paged_decode_attn");
    // what decode_status() needs to find the call's status word
    Ref w(THPVariable_Wrap(ws)), d(THPDevice_New(dev));
    Ref last(Py_BuildValue("(OLLLLO)", w.o, static_cast<long long>(B), static_cast<long long>(Hq),
                           max_seq, static_cast<long long>(L), d.o));
    if (PyObject_SetAttr(self, names._last_decode, last.o) < 0) throw PyError{};
    if (a[7] != Py_None) return Py_NewRef(a[7]);
    return THPVariable_Wrap(out);
}

// paged_chunk(self, q, block_table, seq_lens, max_seq_len, scale, layer)
PyObject* paged_chunk(PyObject* const* a) {
    PyObject* self = a[0];
    at::Tensor q = cuda_tensor(a[1], "q");
    if (!q.is_contiguous()) q = q.contiguous();
    const Pool p(self);
    const int64_t B = q.size(0), q_len = q.size(1), Hq = q.size(2), D = q.size(3);
    const double scale = a[5] == Py_None ? std::pow(static_cast<double>(D), -0.5) : as_double(a[5]);
    const at::Device dev = q.device();
    const at::Tensor bt = as_i32(a[2], "block_table", dev), sl = as_i32(a[3], "seq_lens", dev);
    const long long max_seq = as_int(a[4]);
    const c10::cuda::CUDAGuard guard(dev);
    const at::Tensor out = empty(q.sizes(), q.scalar_type(), dev);
    void* st = stream_of(dev);
    const at::Tensor ws = workspace(Py_None, dev, st, api.ftq_paged_chunk_workspace_bytes(
                                                          B, q_len, Hq, p.hkv, p.d, max_seq));
    uint8_t* base = p.base(a[6]);
    Ref so(PyObject_GetAttr(self, names.signs)), ko(PyObject_GetAttr(self, names.levels_k)),
        vo(PyObject_GetAttr(self, names.levels_v));
    const Table signs(so.o), lk(ko.o), lv(vo.o);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_paged_chunk_attn(
            ptr<void>(q), dtype_code(q.scalar_type()), mptr<void>(out), dtype_code(out.scalar_type()), base,
            p.num_blocks, ptr<int32_t>(bt), bt.size(1), ptr<int32_t>(sl), max_seq, B, q_len, Hq, p.hkv, D,
            p.kb, p.vb, lk.p, lv.p, signs.p, static_cast<float>(scale), mptr<void>(ws), ws.numel(), st);
    }
    check(rc, "ftq_paged_chunk_attn");
    // (the status word lies where a decode call of one sequence has it)
    Ref w(THPVariable_Wrap(ws)), d(THPDevice_New(dev));
    Ref last(Py_BuildValue("(OLLLLO)", w.o, 1ll, static_cast<long long>(Hq), max_seq, 1ll, d.o));
    if (PyObject_SetAttr(self, names._last_decode, last.o) < 0) throw PyError{};
    return THPVariable_Wrap(out);
}

int64_t packed_dim(int64_t d, long long bits) {
    if (bits < 2 || bits > 4)
        raise(PyExc_ValueError, "bits must be 2, 3, or 4, got " + std::to_string(bits));
    return d * bits / 8;
}

// encode(x, signs, boundaries, bits) -> (packed, norms)
PyObject* encode(PyObject* const* a) {
    at::Tensor x = supported(cuda_tensor(a[0], "x"));
    if (!x.is_contiguous()) x = x.contiguous();
    const long long bits = as_int(a[3]);
    const int64_t d = x.size(-1), pd = packed_dim(d, bits), n = d ? x.numel() / d : 0;
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 1);
    const at::Device dev = x.device();
    const Table signs(a[1]), bounds(a[2]);
    const c10::cuda::CUDAGuard guard(dev);
    const at::Tensor norms = empty(shape, at::kHalf, dev);
    shape.push_back(pd);
    const at::Tensor packed = empty(shape, at::kByte, dev);
    void* st = stream_of(dev);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_encode(ptr<void>(x), dtype_code(x.scalar_type()), n, d, d, bits, signs.p, bounds.p,
                            mptr(packed), mptr<uint16_t>(norms), st);
    }
    check(rc, "ftq_encode");
    Ref r0(THPVariable_Wrap(packed)), r1(THPVariable_Wrap(norms));
    return PyTuple_Pack(2, r0.o, r1.o);
}

// decode_dense(packed, norms, levels, signs, bits, head_dim) -> fp32 [..., head_dim]
PyObject* decode_dense(PyObject* const* a) {
    at::Tensor packed = cuda_tensor(a[0], "packed_indices"), norms = tensor(a[1], "norms");
    const long long bits = as_int(a[4]), d = as_int(a[5]);
    const int64_t pd = packed_dim(d, bits);
    if (pd <= 0 || packed.numel() % pd) raise(PyExc_RuntimeError, "packed_indices do not split into rows");
    if (!packed.is_contiguous()) packed = packed.contiguous();
    if (!norms.is_contiguous()) norms = norms.contiguous();
    if (norms.scalar_type() != at::kHalf && norms.scalar_type() != at::kFloat) norms = norms.to(at::kFloat);
    const at::Device dev = packed.device();
    const Table levels(a[2]), signs(a[3]);
    const c10::cuda::CUDAGuard guard(dev);
    std::vector<int64_t> shape(norms.sizes().begin(), norms.sizes().end());
    shape.push_back(d);
    const at::Tensor out = empty(shape, at::kFloat, dev);
    void* st = stream_of(dev);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_decode_dense(ptr(packed), ptr<void>(norms), dtype_code(norms.scalar_type()),
                                  norms.numel(), d, bits, levels.p, signs.p, mptr<float>(out), st);
    }
    check(rc, "ftq_decode_dense");
    return THPVariable_Wrap(out);
}

// rht(x, signs, inverse) -> same shape and dtype
PyObject* rht(PyObject* const* a) {
    const at::Tensor& given = cuda_tensor(a[0], "x");
    at::Tensor x = supported(given);
    if (!x.is_contiguous()) x = x.contiguous();
    const int64_t d = x.size(-1);
    const at::Device dev = x.device();
    const Table signs(a[1]);
    const bool inverse = as_bool(a[2]);
    const c10::cuda::CUDAGuard guard(dev);
    at::Tensor y = empty(x.sizes(), x.scalar_type(), dev);
    void* st = stream_of(dev);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_rht(ptr<void>(x), mptr<void>(y), dtype_code(x.scalar_type()), d ? x.numel() / d : 0, d,
                         signs.p, inverse, st);
    }
    check(rc, "ftq_rht");
    if (y.scalar_type() != given.scalar_type()) y = y.to(given.scalar_type());
    return THPVariable_Wrap(y);
}

// flash_decode(q, k_idx, k_norms, v_idx, v_norms, levels_k, levels_v, signs, scale, bits_k, bits_v,
//              seq_lens, q_is_rotated, out_dtype, workspace) -> out [B, Hq, 1, D]
PyObject* flash_decode(PyObject* const* a) {
    at::Tensor q = supported(cuda_tensor(a[0], "q_rotated"));
    if (q.dim() != 4 || q.size(2) != 1)
        raise(PyExc_ValueError, "flash_decode_compressed handles one query token per sequence");
    if (!q.is_contiguous()) q = q.contiguous();
    auto dense = [](PyObject* o, const char* name) {
        const at::Tensor& t = tensor(o, name);
        return t.is_contiguous() ? t : t.contiguous();
    };
    auto half = [&](PyObject* o, const char* name) {
        at::Tensor t = dense(o, name);
        return t.scalar_type() == at::kHalf ? t : t.to(at::kHalf);
    };
    const at::Tensor ki = dense(a[1], "k_indices"), kn = half(a[2], "k_norms"),
                     vi = dense(a[3], "v_indices"), vn = half(a[4], "v_norms");
    if (ki.dim() != 4) raise(PyExc_ValueError, "k_indices must be [B, Hkv, S, packed]");
    const int64_t B = q.size(0), Hq = q.size(1), d = q.size(3), Hkv = ki.size(1), S = ki.size(2);
    const Table lk(a[5]), lv(a[6]), signs(a[7]);
    const at::Device dev = q.device();
    at::Tensor sl;
    if (a[11] != Py_None) sl = as_i32(a[11], "seq_lens", dev);
    const c10::cuda::CUDAGuard guard(dev);
    at::ScalarType ot = at::kFloat;
    if (a[13] != Py_None) {
        if (!THPDtype_Check(a[13])) raise(PyExc_TypeError, "out_dtype must be a torch.dtype");
        ot = reinterpret_cast<THPDtype*>(a[13])->scalar_type;
    }
    const at::Tensor out = empty(q.sizes(), ot, dev);
    const int oc = out_dtype_code(out);
    void* st = stream_of(dev);
    const at::Tensor ws = workspace(a[14], dev, st, api.ftq_decode_workspace_bytes(B, Hq, Hkv, d, S, 1));
    const double scale = as_double(a[8]);
    const long long bk = as_int(a[9]), bv = as_int(a[10]);
    const bool rotated = as_bool(a[12]);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_flash_decode(ptr<void>(q), dtype_code(q.scalar_type()), rotated, ptr(ki),
                                  ptr<uint16_t>(kn), ptr(vi), ptr<uint16_t>(vn), lk.p, lv.p, signs.p,
                                  static_cast<float>(scale), bk, bv,
                                  sl.defined() ? ptr<int32_t>(sl) : nullptr, B, Hq, Hkv, S, d,
                                  mptr<void>(out), oc, mptr<void>(ws), ws.numel(), st);
    }
    check(rc, "ftq_flash_decode");
    return THPVariable_Wrap(out);
}

// The slot cache as bytes, and its strides (base of layer 0).
struct SlotCache {
    at::Tensor t;
    bool layered;
    int64_t sb, sp, sh, block_size, hkv, num_blocks, layer_stride;
    SlotCache(PyObject* o, bool want_layers, const char* mismatch) {
        t = cuda_tensor(o, "kv_cache");
        if (t.scalar_type() != at::kByte) t = t.view(at::kByte);
        layered = want_layers;
        if (layered != (t.dim() == 5)) raise(PyExc_ValueError, mismatch);
        if (t.dim() != (layered ? 5 : 4) || t.stride(-1) != 1)
            raise(PyExc_ValueError,
                  "kv_cache must be [num_blocks, block_size, num_kv_heads, slot] with a dense last dim");
        sb = t.stride(-4); sp = t.stride(-3); sh = t.stride(-2);
        num_blocks = t.size(-4); block_size = t.size(-3); hkv = t.size(-2);
        layer_stride = layered ? t.stride(0) : 0;
    }
};

// tq_store(key, value, kv_cache, slot_mapping, midpoints, key_bits, value_bits, rotate_in_kernel,
//          v_lloyd_max)
PyObject* tq_store(PyObject* const* a) {
    at::Tensor key = supported(cuda_tensor(a[0], "key"));
    at::Tensor value = tensor(a[1], "value");
    const bool layered = key.dim() == 4;
    const SlotCache c(a[2], layered,
                      "key/value [L, N, Hkv, D] go with a cache [L, num_blocks, block_size, Hkv, slot]");
    const int64_t L = layered ? key.size(0) : 1;
    if (layered && c.t.size(0) != L)
        raise(PyExc_ValueError, "key/value and kv_cache disagree on the number of layers");
    if (value.scalar_type() != key.scalar_type()) value = value.to(key.scalar_type());
    if (key.stride(-1) != 1 || value.strides() != key.strides()) {
        key = key.contiguous();
        value = value.contiguous();
    }
    const at::Device dev = key.device();
    const at::Tensor sm = as_i64(a[3], "slot_mapping", dev);
    const long long kb = as_int(a[5]), vb = as_int(a[6]);
    const int64_t d = key.size(-1);
    const int64_t slot = (kb == 8 ? d : kb == FTQ_TQ_KEY_BITS_MSE8 ? d + 2 : (d * kb + 7) / 8 + 2) +
                         (d * vb + 7) / 8 + 4;
    if (c.t.size(-1) < slot)
        raise(PyExc_ValueError, "kv_cache slots of " + std::to_string(c.t.size(-1)) +
              " bytes are smaller than " + std::to_string(slot));
    const Table mids(kb == 8 ? Py_None : a[4]);
    const bool rotate = as_bool(a[7]), lloyd = as_bool(a[8]);
    const c10::cuda::CUDAGuard guard(dev);
    void* st = stream_of(dev);
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_tq_store_layers(
            ptr<void>(key), ptr<void>(value), dtype_code(key.scalar_type()), key.size(-3), key.size(-2),
            key.size(-1), key.stride(-3), key.stride(-2), kb, vb, rotate, lloyd, mids.p, mptr(c.t), c.sb,
            c.sp, c.sh, c.block_size, ptr<int64_t>(sm), L, layered ? key.stride(0) : 0, c.layer_stride,
            c.num_blocks, st);
    }
    check(rc, "ftq_tq_store_layers");
    Py_RETURN_NONE;
}

// tq_decode(query, kv_cache, block_table, seq_lens, kv_start_offset, centroids, key_bits, value_bits,
//           norm_correction, v_rotate, v_lloyd_max, scale, num_kv_splits, mid_o, output, out_dtype,
//           lse, prefix_output, prefix_lse, head_dim, workspace)
PyObject* tq_decode(PyObject* const* a) {
    at::Tensor q = supported(cuda_tensor(a[0], "query"));
    const bool layered = q.dim() == 4;
    if (!layered && q.dim() != 3) raise(PyExc_ValueError, "query must be [(L,) B, Hq, D]");
    const SlotCache c(a[1], layered,
                      layered ? "a [L, B, Hq, D] query needs a [L, num_blocks, block_size, Hkv, slot] cache"
                              : "kv_cache must be [num_blocks, block_size, num_kv_heads, slot] with a dense last dim");
    const int64_t L = layered ? q.size(0) : 1;
    if (layered && c.t.size(0) != L)
        raise(PyExc_ValueError, "a [L, B, Hq, D] query needs a [L, num_blocks, block_size, Hkv, slot] cache");
    const int64_t B = q.size(-3), hq = q.size(-2), d = q.size(-1), rows = L * B;
    if (d != as_int(a[19]))
        raise(PyExc_ValueError, "query head size " + std::to_string(d) + " does not match the config (" +
              std::to_string(as_int(a[19])) + ")");
    if (!q.is_contiguous()) q = q.contiguous();
    const at::Device dev = q.device();
    const at::Tensor bt = as_i32(a[2], "block_table", dev), sl = as_i32(a[3], "seq_lens", dev);
    if (bt.dim() < 2) raise(PyExc_IndexError, "block_table must be [B, max_blocks]");
    at::Tensor ks, mid, lse, po, pl;
    if (a[4] != Py_None) ks = as_i32(a[4], "kv_start_offset", dev);
    const long long kb = as_int(a[6]), vb = as_int(a[7]), splits = as_int(a[12]);
    const Table cent(kb == 8 ? Py_None : a[5]);
    const c10::cuda::CUDAGuard guard(dev);
    if (a[13] == Py_None) {
        mid = empty({rows, hq, splits, d + 1}, at::kFloat, dev);
    } else {
        mid = tensor(a[13], "mid_o");
        if (mid.numel() != rows * hq * splits * (d + 1) || mid.scalar_type() != at::kFloat || !mid.is_contiguous())
            raise(PyExc_ValueError, "mid_o must be a contiguous fp32 [(L,) B, Hq, num_kv_splits, D+1] tensor");
    }
    at::Tensor out;
    if (a[14] == Py_None) {
        at::ScalarType ot = q.scalar_type();
        if (a[15] != Py_None) {
            if (!THPDtype_Check(a[15])) raise(PyExc_TypeError, "out_dtype must be a torch.dtype");
            ot = reinterpret_cast<THPDtype*>(a[15])->scalar_type;
        }
        out = empty(q.sizes(), ot, dev);
    } else {
        out = tensor(a[14], "output");
        if (out.sizes() != q.sizes() || !out.is_contiguous() || dtype_code(out.scalar_type()) < 0)
            raise(PyExc_ValueError, "output must be a contiguous [(L,) B, Hq, D] tensor of a supported dtype");
    }
    const int oc = out_dtype_code(out);
    if (a[16] != Py_None) {
        lse = tensor(a[16], "lse");
        if (lse.scalar_type() != at::kFloat || !lse.is_contiguous() || lse.numel() != rows * hq || lse.device() != dev)
            raise(PyExc_ValueError, "lse must be a contiguous fp32 [(L,) B, Hq] tensor on the query's device");
    }
    if ((a[17] == Py_None) != (a[18] == Py_None))
        raise(PyExc_ValueError, "prefix_output and prefix_lse go together");
    if (a[17] != Py_None) {
        po = cuda_tensor(a[17], "prefix_output");
        pl = tensor(a[18], "prefix_lse");
        if (po.sizes() != q.sizes() || pl.sizes() != q.sizes().slice(0, q.dim() - 1))
            raise(PyExc_ValueError, "prefix_output must be [(L,) B, Hq, D] and prefix_lse [(L,) B, Hq]");
        po = supported(po).contiguous();
        pl = pl.to(dev, at::kFloat).contiguous();
    }
    const bool nc = as_bool(a[8]), rot = as_bool(a[9]), lloyd = as_bool(a[10]);
    const double scale = as_double(a[11]);
    void* st = stream_of(dev);
    // Scratch of the kernel that streams whole pages: the caller's, or a tensor of the call's own (a captured graph keeps its
    // memory, whatever later calls need).  Where that kernel is not taken nothing is allocated; without memory for it the
    // item kernels run, which need none.
    at::Tensor ws;
    if (a[20] != Py_None) {
        ws = tensor(a[20], "workspace");
        if (ws.device() != dev || !ws.is_contiguous())
            raise(PyExc_ValueError, "workspace must be a contiguous tensor on the query's device");
    } else if (const size_t need = hq > 0 && c.hkv > 0 ? api.ftq_tq_decode_layers_workspace_bytes(
                   dtype_code(q.scalar_type()), B, hq, c.hkv, d, ptr(c.t), c.sb, c.sp, c.sh, c.block_size, bt.size(1), kb, vb,
                   lloyd, splits, L, c.layer_stride) : 0) {
        try {
            ws = empty({static_cast<int64_t>(need)}, at::kByte, dev);
        } catch (const c10::OutOfMemoryError&) {
        }
    }
    int rc;
    {
        NoGil nogil;
        rc = api.ftq_tq_decode_layers_ws(
            ptr<void>(q), dtype_code(q.scalar_type()), B, hq, c.hkv, d, ptr(c.t), c.sb, c.sp, c.sh,
            c.block_size, ptr<int32_t>(bt), bt.size(1), ptr<int32_t>(sl), ks.defined() ? ptr<int32_t>(ks) : nullptr,
            kb, vb, nc, rot, lloyd, cent.p, static_cast<float>(scale), splits, mptr<float>(mid),
            mptr<void>(out), oc, lse.defined() ? mptr<float>(lse) : nullptr,
            po.defined() ? ptr<void>(po) : nullptr, po.defined() ? dtype_code(po.scalar_type()) : 0,
            pl.defined() ? ptr<float>(pl) : nullptr, L, c.layer_stride, c.num_blocks,
            ws.defined() ? mptr<void>(ws) : nullptr, ws.defined() ? ws.nbytes() : 0, st);
    }
    check(rc, "ftq_tq_decode_layers_ws");
    if (a[14] != Py_None) return Py_NewRef(a[14]);
    return THPVariable_Wrap(out);
}

// bind({name: address}, check, get_workspace, workspaces, host_table)
PyObject* bind(PyObject* const* a) {
#define X(name)                                                                     \
    {                                                                               \
        PyObject* v = PyDict_GetItemString(a[0], #name);                            \
        if (!v) raise(PyExc_KeyError, #name);                                       \
        api.name = reinterpret_cast<decltype(api.name)>(PyLong_AsVoidPtr(v));       \
    }
    FTQ_BOUND(X)
#undef X
    g_check = Py_NewRef(a[1]);
    g_get_workspace = Py_NewRef(a[2]);
    g_workspaces = Py_NewRef(a[3]);
    g_host_table = Py_NewRef(a[4]);
    Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject* const*), Py_ssize_t N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    try {
        want_args(n, N, "fused_turboquant_b200._native");
        return F(args);
    } catch (const PyError&) {
        return nullptr;
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

#define FTQ_ENTRY(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FTQ_ENTRY(bind, 5),
    FTQ_ENTRY(paged_store, 5),
    FTQ_ENTRY(paged_decode, 9),
    FTQ_ENTRY(paged_chunk, 7),
    FTQ_ENTRY(encode, 4),
    FTQ_ENTRY(decode_dense, 6),
    FTQ_ENTRY(rht, 3),
    FTQ_ENTRY(flash_decode, 15),
    FTQ_ENTRY(tq_store, 9),
    FTQ_ENTRY(tq_decode, 21),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", "Tensor-level host path over libftq_b200.so.",
                          -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
#define X(name) names.name = PyUnicode_InternFromString(#name);
    FTQ_NAMES(X)
#undef X
    PyObject* m = PyModule_Create(&module_def);
    if (m && PyModule_AddStringConstant(m, "BUILT_FOR", FTQ_BUILT_FOR) < 0) Py_CLEAR(m);
    return m;
}
