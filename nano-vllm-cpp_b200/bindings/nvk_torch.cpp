// CPython binding of the C ABI (include/nvk.h) for torch tensors: argument checks, pointers, sizes and the current stream
// in one native call.
//
// A decode or prefill call of a few rows is bound by the host: through ctypes the 20 to 30 argument objects of one call,
// the per-tensor attribute look-ups and the stream query took about 14 us, more than the kernels they launch.  Here a call
// reads the tensors' fields directly and takes well under a microsecond on top of the launches themselves.  Each function
// takes its arguments by position (the Python wrappers in __init__.py carry names and defaults) and returns how many
// kernels it launched (decode: at least).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

#include "../../include/nvk.h"

namespace {

struct Raised {};   // a Python exception is set

[[noreturn]] void raise(PyObject* type, const char* fmt, const char* name) {
    PyErr_Format(type, fmt, name);
    throw Raised{};
}

void check(int rc) {
    if (rc == NVK_OK) return;
    PyErr_SetString(rc == NVK_ERR_INVALID_ARGUMENT || rc == NVK_ERR_UNSUPPORTED ? PyExc_ValueError : PyExc_RuntimeError, nvk_last_error());
    throw Raised{};
}

// One call of the library, with the interpreter free for other threads meanwhile: a launch blocks while the queue is full, and in a process
// with a thread per rank the one that would launch what the GPU is waiting for must not wait for this one.  (The arguments are
// evaluated before.)
template <typename... P, typename... A> void launch(int (*function)(P...), A... args) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = function(args...);
    Py_END_ALLOW_THREADS
    check(rc);
}

int code(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kHalf: return NVK_F16;
        case at::kBFloat16: return NVK_BF16;
        case at::kFloat: return NVK_F32;
        case at::kInt: return NVK_I32;
        case at::kLong: return NVK_I64;
        case at::kChar: return NVK_I8;
        default: raise(PyExc_KeyError, "%s", c10::toString(t.scalar_type()));
    }
}

const at::Tensor* optional(const char* name, PyObject* o) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "%s must be a tensor", name);
    return &THPVariable_Unpack(o);
}

// A contiguous CUDA tensor, or an exception.
const at::Tensor& cuda(const char* name, PyObject* o) {
    const at::Tensor* t = optional(name, o);
    if (t == nullptr) raise(PyExc_ValueError, "%s must be defined", name);
    if (!t->is_cuda()) raise(PyExc_ValueError, "%s must live on CUDA", name);
    if (!t->is_contiguous()) raise(PyExc_ValueError, "%s must be contiguous", name);
    return *t;
}
const at::Tensor* optional_cuda(const char* name, PyObject* o) { return o == Py_None ? nullptr : &cuda(name, o); }

void* ptr(const at::Tensor& t) { return t.numel() > 0 ? t.data_ptr() : nullptr; }
void* ptr(const at::Tensor* t) { return t != nullptr ? ptr(*t) : nullptr; }
size_t bytes(const at::Tensor* t) { return t != nullptr ? t->nbytes() : 0; }
int64_t numel(const at::Tensor* t) { return t != nullptr ? t->numel() : 0; }
int64_t size(const at::Tensor& t, int64_t d, const char* name) {
    if (d >= t.dim()) raise(PyExc_IndexError, "%s has too few dimensions", name);
    return t.size(d);
}

int64_t integer(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw Raised{};
    return v;
}
float real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Raised{};
    return static_cast<float>(v);
}

struct Index {   // an index tensor: int32 or int64
    const void* p = nullptr;
    int dtype = NVK_I32;
    Index(const char* name, const at::Tensor* t) {
        if (t == nullptr) return;
        if (t->scalar_type() != at::kInt && t->scalar_type() != at::kLong) raise(PyExc_ValueError, "%s must be int32 or int64", name);
        p = ptr(*t);
        dtype = code(*t);
    }
};

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

int64_t cache_blocks(const at::Tensor& cache, int64_t block_size, int64_t kv_heads, int64_t head_dim) {
    const int64_t per = block_size * kv_heads * head_dim;
    if (per == 0) raise(PyExc_ZeroDivisionError, "%s", "block_size, num_kv_heads and head_dim must be positive");
    return cache.numel() / per;
}
int64_t rows_of(const at::Tensor& cache, int64_t row) {
    if (row == 0) raise(PyExc_ZeroDivisionError, "%s", "a cache row must have elements");
    return cache.numel() / row;
}

// (key, value, k_cache, v_cache, slot_mapping)
long store_kvcache(PyObject* const* a) {
    const at::Tensor &key = cuda("key", a[0]), &value = cuda("value", a[1]), &kc = cuda("k_cache", a[2]), &vc = cuda("v_cache", a[3]),
                     &slots = cuda("slot_mapping", a[4]);
    if (key.scalar_type() != value.scalar_type() || key.scalar_type() != kc.scalar_type() || key.scalar_type() != vc.scalar_type())
        raise(PyExc_ValueError, "%s", "key and value must have the same dtype");
    const int64_t n = slots.numel();
    if (n <= 0) raise(PyExc_ValueError, "%s", "slot_mapping must contain at least one element");
    if (key.numel() % n != 0 || key.numel() != value.numel())
        raise(PyExc_ValueError, "%s", "key cannot be flattened by the provided leading count");
    const int64_t row = key.numel() / n;
    const int64_t cache_rows = rows_of(kc, row);
    if (kc.numel() % row != 0 || kc.numel() != vc.numel()) raise(PyExc_ValueError, "%s", "k_cache does not contain an integer number of cache rows");
    launch(nvk_store_kvcache, ptr(key), ptr(value), ptr(kc), ptr(vc), ptr(slots), code(slots), n, row, cache_rows, code(key), stream());
    return 1;
}

// (qkv, positions, q_norm_weight, k_norm_weight, norm_eps, cos_sin_cache, slot_mapping, k_cache, v_cache, num_q_heads, num_kv_heads,
//  head_dim, q_out)
long fused_split_norm_rope_store(PyObject* const* a) {
    const at::Tensor &qkv = cuda("qkv", a[0]), &pos = cuda("positions", a[1]), &table = cuda("cos_sin_cache", a[5]), &kc = cuda("k_cache", a[7]),
                     &vc = cuda("v_cache", a[8]), &q_out = cuda("q_out", a[12]);
    const at::Tensor *qw = optional_cuda("q_norm_weight", a[2]), *kw = optional_cuda("k_norm_weight", a[3]), *slots = optional_cuda("slot_mapping", a[6]);
    const int64_t hq = integer(a[9]), hkv = integer(a[10]), d = integer(a[11]);
    launch(nvk_fused_split_norm_rope_store, ptr(qkv), static_cast<const int32_t*>(ptr(pos)), ptr(qw), ptr(kw), real(a[4]),
                                            static_cast<const float*>(ptr(table)), size(table, 0, "cos_sin_cache"), static_cast<const int32_t*>(ptr(slots)),
                                            ptr(kc), ptr(vc), rows_of(kc, hkv * d), size(qkv, 0, "qkv"), static_cast<int>(hq), static_cast<int>(hkv),
                                            static_cast<int>(d), ptr(q_out), code(qkv), stream());
    return 1;
}

// The tensors that every decode call has: query, caches, context_lens, block_tables, output and the four numbers.
struct Decode {
    const at::Tensor &q, &kc, &vc, &ctx, &bt, &out;
    Index lens, tables;
    int64_t batch, heads, max_blocks, hkv, d, bs, blocks;
    float scale;
    Decode(PyObject* q_, PyObject* kc_, PyObject* vc_, PyObject* ctx_, PyObject* bt_, PyObject* out_, PyObject* hkv_, PyObject* d_, PyObject* bs_,
           PyObject* scale_)
        : q(cuda("query", q_)), kc(cuda("k_cache", kc_)), vc(cuda("v_cache", vc_)), ctx(cuda("context_lens", ctx_)),
          bt(cuda("block_tables", bt_)), out(cuda("output", out_)), lens("context_lens", &ctx), tables("block_tables", &bt),
          batch(size(q, 0, "query")), heads(size(q, 1, "query")), max_blocks(size(bt, 1, "block_tables")), hkv(integer(hkv_)), d(integer(d_)),
          bs(integer(bs_)), blocks(cache_blocks(kc, bs, hkv, d)), scale(real(scale_)) {}
    // At least: contexts of wider tables are always taken in chunks, which a second kernel brings together; narrower ones may be.
    long launches(const at::Tensor* ws) const {
        return ws != nullptr && d == 128 && q.scalar_type() != at::kFloat && heads <= 8 * hkv && bs % 16 == 0 && max_blocks * bs > 4096 ? 2 : 1;
    }
};

// (query, k_cache, v_cache, context_lens, block_tables, num_kv_heads, head_dim, block_size, scale, output, workspace)
long decode(PyObject* const* a) {
    const Decode x(a[0], a[1], a[2], a[3], a[4], a[9], a[5], a[6], a[7], a[8]);
    const at::Tensor* ws = optional("workspace", a[10]);
    launch(nvk_decode_attention_paged, ptr(x.q), ptr(x.kc), ptr(x.vc), x.lens.p, x.lens.dtype, x.tables.p, x.tables.dtype, x.batch, x.max_blocks,
                                       x.blocks, static_cast<int>(x.heads), static_cast<int>(x.hkv), static_cast<int>(x.d), static_cast<int>(x.bs),
                                       x.scale, ptr(x.out), code(x.q), ptr(ws), bytes(ws), stream());
    return x.launches(ws);
}

// the same without a workspace
long decode_static(PyObject* const* a) {
    const Decode x(a[0], a[1], a[2], a[3], a[4], a[9], a[5], a[6], a[7], a[8]);
    launch(nvk_decode_attention_paged_static, ptr(x.q), ptr(x.kc), ptr(x.vc), x.lens.p, x.lens.dtype, x.tables.p, x.tables.dtype, x.batch, x.max_blocks,
                                              x.blocks, static_cast<int>(x.heads), static_cast<int>(x.hkv), static_cast<int>(x.d),
                                              static_cast<int>(x.bs), x.scale, ptr(x.out), code(x.q), stream());
    return 2;
}

// (query, k_cache, v_cache, k_scale, v_scale, context_lens, block_tables, num_kv_heads, head_dim, block_size, scale, output, workspace)
template <bool FP8> long decode8(PyObject* const* a) {
    const Decode x(a[0], a[1], a[2], a[5], a[6], a[11], a[7], a[8], a[9], a[10]);
    const at::Tensor &ks = cuda("k_scale", a[3]), &vs = cuda("v_scale", a[4]);
    const at::Tensor* ws = optional("workspace", a[12]);
    launch(FP8 ? nvk_decode_attention_paged_fp8 : nvk_decode_attention_paged_int8,
        ptr(x.q), ptr(x.kc), ptr(x.vc), ptr(ks), ptr(vs), x.lens.p, x.lens.dtype, x.tables.p, x.tables.dtype, x.batch, x.max_blocks, x.blocks,
        static_cast<int>(x.heads), static_cast<int>(x.hkv), static_cast<int>(x.d), static_cast<int>(x.bs), x.scale, ptr(x.out), code(x.q), ptr(ws),
        bytes(ws), stream());
    return x.launches(ws);
}

// (key, value, k_cache, v_cache, k_scale, v_scale, slot_mapping)
template <bool FP8> long store8(PyObject* const* a) {
    const at::Tensor &key = cuda("key", a[0]), &value = cuda("value", a[1]), &kc = cuda("k_cache", a[2]), &vc = cuda("v_cache", a[3]),
                     &ks = cuda("k_scale", a[4]), &vs = cuda("v_scale", a[5]), &slots = cuda("slot_mapping", a[6]);
    if (FP8) {
        if (kc.element_size() != 1 || vc.element_size() != 1) raise(PyExc_ValueError, "%s", "store_kvcache_fp8 requires one-byte caches");
    } else if (kc.scalar_type() != at::kChar || vc.scalar_type() != at::kChar) {
        raise(PyExc_ValueError, "%s", "store_kvcache_int8 requires int8 caches");
    }
    if (ks.scalar_type() != at::kHalf || vs.scalar_type() != at::kHalf)
        raise(PyExc_ValueError, "store_kvcache_%s requires float16 scales", FP8 ? "fp8" : "int8");
    if (key.dim() != 3) raise(PyExc_ValueError, "key must be rank-3 for %s store", FP8 ? "the fp8" : "int8");
    if (slots.element_size() != 4) raise(PyExc_ValueError, "%s", "slot_mapping must be int32");
    const int64_t hkv = key.size(1), d = key.size(2);
    launch(FP8 ? nvk_store_kvcache_fp8 : nvk_store_kvcache_int8, ptr(key), ptr(value), ptr(kc), ptr(vc), ptr(ks), ptr(vs),
                                                                   static_cast<const int32_t*>(ptr(slots)), slots.numel(), static_cast<int>(hkv),
                                                                   static_cast<int>(d), rows_of(kc, hkv * d), code(key), stream());
    return 1;
}

// (query, key, value, k_cache, v_cache, cu_q, cu_k, block_tables, num_kv_heads, head_dim, block_size, scale, output, max_seqlen_q)
long prefill(PyObject* const* a) {
    const at::Tensor &q = cuda("query", a[0]), &out = cuda("output", a[12]);
    const at::Tensor *cu_q = optional("cu_seqlens_q", a[5]), *cu_k = optional("cu_seqlens_k", a[6]), *bt = optional_cuda("block_tables", a[7]);
    const at::Tensor *k = nullptr, *v = nullptr, *kc = nullptr, *vc = nullptr;
    if (bt != nullptr) {
        kc = &cuda("k_cache", a[3]); vc = &cuda("v_cache", a[4]);
    } else {
        k = &cuda("key", a[1]); v = &cuda("value", a[2]);
    }
    const Index iq("cu_seqlens_q", cu_q), ik("cu_seqlens_k", cu_k), it("block_tables", bt);
    const int64_t hkv = integer(a[8]), d = integer(a[9]), bs = integer(a[10]);
    launch(nvk_prefill_attention_varlen, ptr(q), ptr(k), ptr(v), ptr(kc), ptr(vc), iq.p, iq.dtype, ik.p, ik.dtype, it.p, it.dtype,
                                         cu_q != nullptr ? cu_q->numel() - 1 : 1, size(q, 0, "query"), k != nullptr ? size(*k, 0, "key") : 0,
                                         bt != nullptr ? size(*bt, 1, "block_tables") : 0, kc != nullptr ? cache_blocks(*kc, bs, hkv, d) : 0,
                                         static_cast<int>(integer(a[13])), static_cast<int>(size(q, 1, "query")), static_cast<int>(hkv),
                                         static_cast<int>(d), static_cast<int>(bs), real(a[11]), ptr(out), code(q), stream());
    return 1;
}

// (p_query, cu_seqlens_q, p_key, p_value, cu_seqlens_k, p_block_tables, p_output, d_query, context_lens, d_block_tables, d_output, k_cache,
//  v_cache, num_kv_heads, head_dim, block_size, scale, workspace, prefill_blocks)
long mixed_step(PyObject* const* a) {
    const at::Tensor &pq = cuda("p_query", a[0]), &po = cuda("p_output", a[6]), &ws = cuda("workspace", a[17]);
    const Decode x(a[7], a[11], a[12], a[8], a[9], a[10], a[13], a[14], a[15], a[16]);
    const at::Tensor *cu_q = optional("cu_seqlens_q", a[1]), *pk = optional("p_key", a[2]), *pv = optional("p_value", a[3]),
                     *cu_k = optional("cu_seqlens_k", a[4]), *pt = optional("p_block_tables", a[5]);
    const Index iq("cu_seqlens_q", cu_q), ik("cu_seqlens_k", cu_k), it("p_block_tables", pt);
    launch(nvk_attention_mixed_step, ptr(pq), ptr(pk), ptr(pv), ptr(x.kc), ptr(x.vc), iq.p, iq.dtype, ik.p, ik.dtype, it.p, it.dtype,
                                     cu_q != nullptr ? cu_q->numel() - 1 : 1, size(pq, 0, "p_query"), pk != nullptr ? size(*pk, 0, "p_key") : 0,
                                     pt != nullptr ? size(*pt, 1, "p_block_tables") : 0, 0, ptr(po), ptr(x.q), x.lens.p, x.lens.dtype, x.tables.p,
                                     x.tables.dtype, x.batch, x.max_blocks, ptr(x.out), x.blocks, static_cast<int>(size(pq, 1, "p_query")),
                                     static_cast<int>(x.hkv), static_cast<int>(x.d), static_cast<int>(x.bs), x.scale, code(pq), ptr(ws), ws.nbytes(),
                                     static_cast<int>(integer(a[18])), stream());
    return 2;
}

// (x, weight, out)
long linear(PyObject* const* a) {
    const at::Tensor &x = cuda("x", a[0]), &w = cuda("weight", a[1]), &out = cuda("out", a[2]);
    launch(nvk_linear, ptr(x), ptr(w), ptr(out), size(x, 0, "x"), size(w, 0, "weight"), size(w, 1, "weight"), code(x), stream());
    return 1;
}

// (x, qkv_weight, positions, q_norm_weight, k_norm_weight, norm_eps, cos_sin_cache, slot_mapping, k_cache, v_cache, num_q_heads, num_kv_heads,
//  head_dim, q_out)
long qkv_linear(PyObject* const* a) {
    const at::Tensor &x = cuda("x", a[0]), &w = cuda("qkv_weight", a[1]), &pos = cuda("positions", a[2]), &table = cuda("cos_sin_cache", a[6]),
                     &kc = cuda("k_cache", a[8]), &vc = cuda("v_cache", a[9]), &q_out = cuda("q_out", a[13]);
    const at::Tensor *qw = optional("q_norm_weight", a[3]), *kw = optional("k_norm_weight", a[4]), *slots = optional("slot_mapping", a[7]);
    const int64_t hq = integer(a[10]), hkv = integer(a[11]), d = integer(a[12]);
    launch(nvk_qkv_linear_norm_rope_store, ptr(x), ptr(w), size(x, 0, "x"), size(x, 1, "x"), static_cast<const int32_t*>(ptr(pos)), ptr(qw), ptr(kw),
                                           real(a[5]), static_cast<const float*>(ptr(table)), size(table, 0, "cos_sin_cache"),
                                           static_cast<const int32_t*>(ptr(slots)), ptr(kc), ptr(vc), rows_of(kc, hkv * d), static_cast<int>(hq),
                                           static_cast<int>(hkv), static_cast<int>(d), ptr(q_out), code(x), stream());
    return 1;
}

// One METH_FASTCALL entry: argument count, C++ exceptions to Python ones.
template <long (*F)(PyObject* const*), Py_ssize_t N> PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != N) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", N, n);
        return nullptr;
    }
    try {
        return PyLong_FromLong(F(args));
    } catch (const Raised&) {
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

template <long (*F)(PyObject* const*), Py_ssize_t N> PyMethodDef method(const char* name) {
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(call<F, N>)), METH_FASTCALL, nullptr};
}

PyMethodDef methods[] = {
    method<store_kvcache, 5>("store_kvcache"),
    method<fused_split_norm_rope_store, 13>("fused_split_norm_rope_store"),
    method<decode, 11>("decode"),
    method<decode_static, 10>("decode_static"),
    method<decode8<false>, 13>("decode_int8"),
    method<decode8<true>, 13>("decode_fp8"),
    method<store8<false>, 7>("store_int8"),
    method<store8<true>, 7>("store_fp8"),
    method<prefill, 14>("prefill"),
    method<mixed_step, 19>("mixed_step"),
    method<linear, 3>("linear"),
    method<qkv_linear, 14>("qkv_linear"),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "nvk_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_nvk_torch(void) { return PyModule_Create(&module); }
