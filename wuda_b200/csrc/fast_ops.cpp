// The operators' way from Python to the C ABI without the interpreter in between: argument checks, output allocation, the
// current stream and the launch in one native call.  A call of an operator spends its host time on twenty attribute
// reads, two or three allocations and a foreign-function call with a dozen arguments; the launch itself is 3 us of it.
// Host time per call, one token, before -> after: rmsnorm_quant 12.4 -> 5.3 us, rope_quant 11.1 -> 4.4, act_quant 18.6 -> 6.4,
// fp8_gemm 11.2 -> 6.4, topk 6.7 -> 2.2; norm + RoPE quantisation of 256 tokens, plain calls, 24.4 -> 13.1 us.
//
// Every function takes the arguments of the Python function of its name (ops.py), all positional, and either performs the
// call or returns None, having done nothing: for arguments it does not know (another type of tensor, modes that
// intercept calls, a scratch that has to grow, a stream under capture where scratch is involved) and for arguments that the
// operator refuses.  The Python function then goes on by itself, so what is refused, and how, is said in one place.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/wuda_b200.h"

namespace {

using at::ScalarType;
using at::Tensor;

#define WUDA_ENTRIES(X)                                                                                              \
    X(wuda_mqa_logits_fp8) X(wuda_mqa_logits_fp4) X(wuda_topk) X(wuda_rmsnorm_quant_fp8) X(wuda_rope_quant_fp8)       \
    X(wuda_gemm_fp8_scratch_bytes) X(wuda_gemm_bf16_scratch_bytes) X(wuda_gemm_nvfp4_scratch_bytes)                   \
    X(wuda_gemm_fp8_blockscaled) X(wuda_gemm_fp8_blockscaled_pow2) X(wuda_gemm_fp8_fp4_pow2) X(wuda_gemm_bf16)        \
    X(wuda_gemm_nvfp4) X(wuda_sparse_mla_workspace_bytes) X(wuda_sparse_mla_decode)

struct Entries {
#define X(name) decltype(&::name) name = nullptr;
    WUDA_ENTRIES(X)
#undef X
} entries;

// An argument list that cannot be served here.
struct Pass {};

void need(bool ok) {
    if (!ok) throw Pass{};
}

// Nothing that would see or change the calls the Python functions make: no tracing, function or dispatch mode.
void need_plain_mode() {
    need((c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set).empty() &&
         !at::impl::torch_function_mode_enabled() && !c10::impl::TorchDispatchModeTLS::any_modes_set());
}

const Tensor& tensor(PyObject* o) {
    need(THPVariable_CheckExact(o));
    return THPVariable_Unpack(o);
}
const Tensor& cuda_tensor(PyObject* o) {
    const Tensor& t = tensor(o);
    need(t.is_cuda());
    return t;
}
const Tensor& dense(PyObject* o, ScalarType type) {
    const Tensor& t = cuda_tensor(o);
    need(t.scalar_type() == type && t.is_contiguous());
    return t;
}
void* address(PyObject* o) { return o == Py_None ? nullptr : tensor(o).data_ptr(); }
int32_t* status_of(PyObject* o) { return static_cast<int32_t*>(address(o)); }

int64_t integer(PyObject* o) {
    need(PyLong_Check(o));
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        throw Pass{};
    }
    return v;
}
int int32(int64_t v) {
    need(v >= INT32_MIN && v <= INT32_MAX);
    return static_cast<int>(v);
}
double real(PyObject* o) {
    need(PyFloat_Check(o) || PyLong_CheckExact(o));
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) {
        PyErr_Clear();
        throw Pass{};
    }
    return v;
}
bool truth(PyObject* o) {
    need(PyBool_Check(o));
    return o == Py_True;
}

Tensor fresh(at::IntArrayRef sizes, ScalarType type, const Tensor& like) {
    return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device()));
}
std::vector<int64_t> with_last(const Tensor& t, int64_t last) {
    std::vector<int64_t> s(t.sizes().begin(), t.sizes().end());
    s.back() = last;
    return s;
}

void* current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// The library's call, without the interpreter lock as a foreign-function call makes it; a refusal is told by the caller's
// own call of the same entry.
template <typename F, typename... Args>
void call(F* f, Args... args) {
    int st;
    Py_BEGIN_ALLOW_THREADS st = f(args...);
    Py_END_ALLOW_THREADS need(st == WUDA_OK);
}

// The eager scratch of (device, stream) as scratch.py keeps it, held until the launch.
struct Scratch {
    PyObject* held = nullptr;
    void* at = nullptr;
    int64_t bytes = 0;
    Scratch(PyObject* streams, const Tensor& on, void* stream, int64_t wanted) {
        need(wanted >= 0 && PyDict_CheckExact(streams) &&
             c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None);
        PyObject* key = Py_BuildValue("(iK)", static_cast<int>(on.get_device()),
                                      static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)));
        if (!key) {
            PyErr_Clear();
            throw Pass{};
        }
        held = PyDict_GetItem(streams, key);      // borrowed
        Py_DECREF(key);
        need(held && PyTuple_CheckExact(held) && PyTuple_GET_SIZE(held) == 4 && PyTuple_GET_ITEM(held, 2) == Py_None);
        at = PyLong_AsVoidPtr(PyTuple_GET_ITEM(held, 0));
        bytes = PyLong_AsLongLong(PyTuple_GET_ITEM(held, 1));
        if (PyErr_Occurred()) PyErr_Clear(), bytes = -1;
        need(bytes >= wanted);
        Py_INCREF(held);
    }
    ~Scratch() { Py_XDECREF(held); }
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
};

PyObject* same(PyObject* o) {
    Py_INCREF(o);
    return o;
}

// ---------------------------------------------------------------- indexer
// q, kv_cache, weights, context_lens, block_table, logits, kv_entries_per_block, kv_block_stride_bytes, next_n, status_word
PyObject* mqa_logits_fp8(PyObject* const* a) {
    const Tensor& q = dense(a[0], ScalarType::Float8_e4m3fn);
    need(q.dim() == 3 && q.size(1) == 64 && q.size(2) == 128);
    const int64_t rows = q.size(0), next_n = integer(a[8]);
    need(next_n >= 1 && rows % next_n == 0);
    const int64_t batch = rows / next_n;
    const Tensor& kv = dense(a[1], ScalarType::Byte);
    const Tensor& w = dense(a[2], ScalarType::Float);
    const Tensor& lens = dense(a[3], ScalarType::Int);
    const Tensor& table = dense(a[4], ScalarType::Int);
    const Tensor& logits = cuda_tensor(a[5]);
    need(w.dim() == 2 && w.size(0) == rows && w.size(1) == 64 && lens.numel() == rows && table.dim() == 2 && table.size(0) == batch &&
         logits.scalar_type() == ScalarType::Float && logits.dim() == 2 && logits.size(0) >= rows && logits.stride(1) == 1 && kv.dim() == 2);
    int64_t stride = integer(a[7]);
    if (stride == 0) stride = kv.size(1);
    need(kv.size(1) == stride);
    call(entries.wuda_mqa_logits_fp8, q.data_ptr(), kv.data_ptr(), static_cast<const float*>(w.data_ptr()),
         static_cast<const int32_t*>(lens.data_ptr()), static_cast<const int32_t*>(table.data_ptr()),
         static_cast<float*>(logits.data_ptr()), int32(batch), int32(next_n), int32(kv.size(0)), int32(integer(a[6])), stride,
         int32(table.size(1)), logits.stride(0), status_of(a[9]), current_stream());
    return same(a[5]);
}

// q, sf_q, kv_cache, weights, context_lens, block_table, logits, max_context_len, kv_entries_per_block, kv_block_stride_bytes,
// status_word
PyObject* mqa_logits_fp4(PyObject* const* a) {
    const Tensor& q = cuda_tensor(a[0]);
    need(q.is_contiguous() && q.element_size() == 1 && q.dim() == 3 && q.size(1) == 64 && q.size(2) == 64);
    const int64_t b = q.size(0);
    const Tensor& sf = dense(a[1], ScalarType::Int);
    const Tensor& kv = dense(a[2], ScalarType::Byte);
    const Tensor& w = dense(a[3], ScalarType::Float);
    const Tensor& lens = dense(a[4], ScalarType::Int);
    const Tensor& table = cuda_tensor(a[5]);
    const Tensor& logits = cuda_tensor(a[6]);
    const int64_t entries_per_block = integer(a[8]), stride = integer(a[9]);
    need(sf.numel() == b * 64 && kv.dim() == 2 && (stride == 0 || stride == kv.size(1)) && w.numel() == b * 64 && lens.numel() == b &&
         table.scalar_type() == ScalarType::Int && table.dim() == 2 && table.size(0) == b && table.stride(1) == 1 &&
         logits.scalar_type() == ScalarType::Float && logits.dim() == 2 && logits.size(0) >= b && logits.stride(1) == 1);
    const int64_t most = a[7] == Py_None ? std::min(logits.size(1), table.size(1) * entries_per_block) : integer(a[7]);
    need(most <= logits.size(1));
    call(entries.wuda_mqa_logits_fp4, q.data_ptr(), static_cast<const int32_t*>(sf.data_ptr()), kv.data_ptr(),
         static_cast<const float*>(w.data_ptr()), static_cast<const int32_t*>(lens.data_ptr()),
         static_cast<const int32_t*>(table.data_ptr()), static_cast<float*>(logits.data_ptr()), int32(b), int32(most), int32(kv.size(0)),
         int32(entries_per_block), kv.size(1), int32(b > 1 ? table.stride(0) : table.size(1)),
         logits.size(0) > 1 ? logits.stride(0) : logits.size(1), status_of(a[10]), current_stream());
    return same(a[6]);
}

// scores, seq_lens, page_table, page_indices, page_size, raw_indices, rows_per_table_row
PyObject* topk(PyObject* const* a) {
    const Tensor& scores = cuda_tensor(a[0]);
    need(scores.scalar_type() == ScalarType::Float && scores.dim() == 2 && scores.stride(1) == 1);
    const int64_t rows = scores.size(0), per = integer(a[6]);
    const Tensor& lens = dense(a[1], ScalarType::Int);
    const Tensor& table = dense(a[2], ScalarType::Int);
    const Tensor& out = dense(a[3], ScalarType::Int);
    need(lens.numel() == rows && table.dim() == 2 && table.size(0) * per == rows && out.dim() == 2 && out.size(0) == rows);
    void* raw = nullptr;
    if (a[5] != Py_None) {
        const Tensor& r = dense(a[5], ScalarType::Int);
        need(r.sizes() == out.sizes());
        raw = r.data_ptr();
    }
    call(entries.wuda_topk, static_cast<const float*>(scores.data_ptr()), static_cast<const int32_t*>(lens.data_ptr()),
         static_cast<const int32_t*>(table.data_ptr()), static_cast<int32_t*>(out.data_ptr()), static_cast<int32_t*>(raw), int32(rows),
         scores.stride(0), table.stride(0), int32(per), int32(out.size(1)), int32(integer(a[4])), current_stream());
    return same(a[3]);
}

// ---------------------------------------------------------------- quantisation
PyObject* triple(const Tensor* y16, const Tensor* y8, const Tensor* sc) {
    PyObject* t = PyTuple_New(3);
    if (!t) return nullptr;
    int i = 0;
    for (const Tensor* v : {y16, y8, sc}) PyTuple_SET_ITEM(t, i++, v && v->defined() ? THPVariable_Wrap(*v) : same(Py_None));
    return t;
}

// x, gamma, eps, quant, scale_fmt, return_bf16
PyObject* rmsnorm_quant(PyObject* const* a) {
    const Tensor& x = cuda_tensor(a[0]);
    need(x.scalar_type() == ScalarType::BFloat16 && x.dim() == 2 && x.stride(1) == 1);
    const int64_t rows = x.size(0), dim = x.size(1);
    const float eps = static_cast<float>(real(a[2]));
    const void* gamma = nullptr;
    int gamma_bf16 = 0;
    if (a[1] != Py_None) {
        const Tensor& g = cuda_tensor(a[1]);
        gamma_bf16 = g.scalar_type() == ScalarType::BFloat16;
        need(g.is_contiguous() && g.numel() == dim && (gamma_bf16 || g.scalar_type() == ScalarType::Float));
        gamma = g.data_ptr();
    }
    const bool quant = truth(a[3]), bf16 = truth(a[5]);
    Tensor y16, y8, sc;
    if (bf16) y16 = fresh({rows, dim}, ScalarType::BFloat16, x);
    if (quant) y8 = fresh({rows, dim}, ScalarType::Float8_e4m3fn, x), sc = fresh({rows, dim / 128}, ScalarType::Float, x);
    call(entries.wuda_rmsnorm_quant_fp8, x.data_ptr(), x.stride(0), gamma, gamma_bf16, eps, bf16 ? y16.data_ptr() : nullptr,
         quant ? y8.data_ptr() : nullptr, quant ? static_cast<float*>(sc.data_ptr()) : nullptr, int32(rows), int32(dim),
         a[4] == Py_None ? 0 : 1, current_stream());
    return triple(&y16, &y8, &sc);
}

// x, scale_fmt (block_size 128)
PyObject* act_quant(PyObject* const* a) {
    const Tensor& x = dense(a[0], ScalarType::BFloat16);
    need(x.dim() >= 1 && x.numel() > 0);
    const int64_t dim = x.size(-1), rows = x.numel() / dim;
    const Tensor y8 = fresh(x.sizes(), ScalarType::Float8_e4m3fn, x), sc = fresh(with_last(x, dim / 128), ScalarType::Float, x);
    call(entries.wuda_rmsnorm_quant_fp8, x.data_ptr(), dim, nullptr, 0, 1e-6f, nullptr, y8.data_ptr(), static_cast<float*>(sc.data_ptr()),
         int32(rows), int32(dim), a[1] == Py_None ? 0 : 1, current_stream());
    PyObject* t = PyTuple_New(2);
    if (!t) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(y8));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(sc));
    return t;
}

// x, positions, cos_table, sin_table, rope_dim, inverse, quant, scale_fmt, return_bf16
PyObject* rope_quant(PyObject* const* a) {
    const Tensor& x = dense(a[0], ScalarType::BFloat16);
    need(x.dim() == 3);
    const int64_t tokens = x.size(0), heads = x.size(1), head_dim = x.size(2), rope_dim = integer(a[4]), width = heads * head_dim;
    const Tensor& pos = dense(a[1], ScalarType::Long);
    const Tensor& cos = dense(a[2], ScalarType::Float);
    const Tensor& sin = dense(a[3], ScalarType::Float);
    need(pos.numel() == tokens && rope_dim >= 0 && cos.dim() == 2 && cos.size(1) == rope_dim / 2 && sin.sizes() == cos.sizes());
    const bool inverse = truth(a[5]), quant = truth(a[6]), bf16 = truth(a[8]);
    Tensor y16, y8, sc;
    if (bf16) y16 = at::empty_like(x);
    if (quant) y8 = fresh({tokens, width}, ScalarType::Float8_e4m3fn, x), sc = fresh({tokens, width / 128}, ScalarType::Float, x);
    call(entries.wuda_rope_quant_fp8, x.data_ptr(), static_cast<const int64_t*>(pos.data_ptr()), static_cast<const float*>(cos.data_ptr()),
         static_cast<const float*>(sin.data_ptr()), bf16 ? y16.data_ptr() : nullptr, quant ? y8.data_ptr() : nullptr,
         quant ? static_cast<float*>(sc.data_ptr()) : nullptr, int32(tokens), int32(heads), int32(head_dim), int32(rope_dim),
         int32(cos.size(0)), static_cast<int>(inverse), a[7] == Py_None ? 0 : 1, current_stream());
    return triple(&y16, &y8, &sc);
}

// ---------------------------------------------------------------- GEMMs
// Scales that are not fp32 (exponent bytes) are the Python functions' to convert: said without an exception, which costs 2.4 us of such a call's
// 41 (fp8_gemm) or 26 (fp4_gemm).
bool fp32_scales(PyObject* o) { return THPVariable_CheckExact(o) && THPVariable_Unpack(o).scalar_type() == ScalarType::Float; }

// C of [.., n] for A of [.., k]; a given one is taken as the Python function takes it
PyObject* result(PyObject* given, const Tensor& made) { return given == Py_None ? THPVariable_Wrap(made) : same(given); }

// a, a_s, b, b_s, out, status_word, pow2_scales, streams
PyObject* fp8_gemm(PyObject* const* p) {
    if (!fp32_scales(p[1]) || !fp32_scales(p[3])) return same(Py_None);
    const Tensor& a = dense(p[0], ScalarType::Float8_e4m3fn);
    const Tensor& a_s = dense(p[1], ScalarType::Float);
    const Tensor& b = dense(p[2], ScalarType::Float8_e4m3fn);
    const Tensor& b_s = dense(p[3], ScalarType::Float);
    need(a.dim() >= 1 && b.dim() == 2 && a.size(-1) > 0);
    const int64_t k = a.size(-1), m = a.numel() / k, n = b.size(0);
    need(b.size(1) == k && a_s.numel() == m * (k / 128) && b_s.dim() == 2 && b_s.size(0) == (n + 127) / 128 && b_s.size(1) == k / 128);
    void* stream = current_stream();
    const Scratch scratch(p[7], a, stream, entries.wuda_gemm_fp8_scratch_bytes(int32(m), int32(n)));
    Tensor made;
    if (p[4] == Py_None) made = fresh(with_last(a, n), ScalarType::BFloat16, a);
    call(truth(p[6]) ? entries.wuda_gemm_fp8_blockscaled_pow2 : entries.wuda_gemm_fp8_blockscaled, a.data_ptr(),
         static_cast<const float*>(a_s.data_ptr()), b.data_ptr(), static_cast<const float*>(b_s.data_ptr()),
         made.defined() ? made.data_ptr() : address(p[4]), int32(m), int32(n), int32(k), scratch.at, scratch.bytes, status_of(p[5]), stream);
    return result(p[4], made);
}

// a, a_s, b, b_s, out, status_word, streams
PyObject* fp4_gemm(PyObject* const* p) {
    if (!fp32_scales(p[1])) return same(Py_None);
    const Tensor& a = dense(p[0], ScalarType::Float8_e4m3fn);
    const Tensor& a_s = dense(p[1], ScalarType::Float);
    const Tensor& b = cuda_tensor(p[2]);
    const Tensor& b_s = cuda_tensor(p[3]);
    need(a.dim() >= 1 && a.size(-1) > 0 && b.is_contiguous() && b.element_size() == 1 && b.dim() == 2);
    const int64_t k = a.size(-1), m = a.numel() / k, n = b.size(0);
    need(b.size(1) * 2 == k && k % 128 == 0 && a_s.numel() == m * (k / 128) && b_s.is_contiguous() && b_s.element_size() == 1 &&
         b_s.dim() == 2 && b_s.size(0) == n && b_s.size(1) == k / 32);
    void* stream = current_stream();
    const Scratch scratch(p[6], a, stream, entries.wuda_gemm_fp8_scratch_bytes(int32(m), int32(n)));
    Tensor made;
    if (p[4] == Py_None) made = fresh(with_last(a, n), ScalarType::BFloat16, a);
    call(entries.wuda_gemm_fp8_fp4_pow2, a.data_ptr(), static_cast<const float*>(a_s.data_ptr()), b.data_ptr(),
         static_cast<const uint8_t*>(b_s.data_ptr()), made.defined() ? made.data_ptr() : address(p[4]), int32(m), int32(n), int32(k),
         scratch.at, scratch.bytes, status_of(p[5]), stream);
    return result(p[4], made);
}

// a, w, out, out_dtype, status_word, streams
PyObject* bf16_gemm(PyObject* const* p) {
    const Tensor& a = dense(p[0], ScalarType::BFloat16);
    const Tensor& w = dense(p[1], ScalarType::BFloat16);
    need(a.dim() >= 1 && a.size(-1) > 0 && w.dim() == 2);
    const int64_t k = a.size(-1), m = a.numel() / k, n = w.size(0);
    need(w.size(1) == k);
    void* stream = current_stream();
    const Scratch scratch(p[5], a, stream, entries.wuda_gemm_bf16_scratch_bytes(int32(m), int32(n)));
    Tensor made;
    if (p[2] == Py_None) {
        need(THPDtype_Check(p[3]));
        made = fresh(with_last(a, n), reinterpret_cast<THPDtype*>(p[3])->scalar_type, a);
    }
    const Tensor& c = made.defined() ? made : tensor(p[2]);
    need(c.is_contiguous() && c.numel() == m * n && (c.scalar_type() == ScalarType::BFloat16 || c.scalar_type() == ScalarType::Float));
    call(entries.wuda_gemm_bf16, a.data_ptr(), w.data_ptr(), c.data_ptr(), static_cast<int>(c.scalar_type() == ScalarType::Float), int32(m),
         int32(n), int32(k), scratch.at, scratch.bytes, status_of(p[4]), stream);
    return result(p[2], made);
}

// a, a_sf_packed, a_global_scale, w, w_sf_packed, w_global_scale, out, status_word, streams
PyObject* nvfp4_gemm(PyObject* const* p) {
    const Tensor& a = dense(p[0], ScalarType::Byte);
    const Tensor& w = dense(p[3], ScalarType::Byte);
    need(a.dim() == 2 && w.dim() == 2 && w.size(1) == a.size(1));
    const int64_t m = a.size(0), k = a.size(1) * 2, n = w.size(0);
    const Tensor& a_sf = cuda_tensor(p[1]);
    const Tensor& w_sf = cuda_tensor(p[4]);
    need(a_sf.scalar_type() == ScalarType::Byte && a_sf.numel() == (m + 127) / 128 * 128 * (k / 16) && w_sf.scalar_type() == ScalarType::Byte &&
         w_sf.numel() == (n + 127) / 128 * 128 * (k / 16));
    const float a_gs = static_cast<float>(real(p[2])), w_gs = static_cast<float>(real(p[5]));
    void* stream = current_stream();
    const Scratch scratch(p[8], a, stream, entries.wuda_gemm_nvfp4_scratch_bytes(int32(m), int32(n)));
    Tensor made;
    if (p[6] == Py_None) made = fresh({m, n}, ScalarType::BFloat16, a);
    call(entries.wuda_gemm_nvfp4, a.data_ptr(), a_sf.data_ptr(), a_gs, w.data_ptr(), w_sf.data_ptr(), w_gs,
         made.defined() ? made.data_ptr() : address(p[6]), int32(m), int32(n), int32(k), scratch.at, scratch.bytes, status_of(p[7]), stream);
    return result(p[6], made);
}

// ---------------------------------------------------------------- attention
// q, (cache, indices, lengths) of the window and of the compressed pool, attn_sink, softmax_scale, out, status_word, split, streams
PyObject* sparse_mla_decode(PyObject* const* p) {
    const Tensor& q = dense(p[0], ScalarType::BFloat16);
    need(q.dim() == 3 && q.size(2) == 512 && q.size(0) >= 1);
    wuda_sparse_mla_args a = {};
    const int64_t batch = q.size(0), heads = q.size(1);
    a.q = q.data_ptr(), a.batch = int32(batch), a.heads = int32(heads);
    a.softmax_scale = static_cast<float>(p[8] == Py_None ? 1.0 / std::sqrt(512.0) : real(p[8]));
    struct Pool {
        const void* data;
        int64_t stride;
        const int32_t *indices, *lengths;
        int32_t pages, entries, capacity;
    };
    const auto pool = [&](PyObject* const* o) -> Pool {
        if (o[0] == Py_None) return {};
        const Tensor& cache = cuda_tensor(o[0]);
        const Tensor& idx = dense(o[1], ScalarType::Int);
        const Tensor& lens = dense(o[2], ScalarType::Int);
        need(cache.element_size() == 1 && cache.dim() == 4 && cache.size(3) == 584 && cache.stride(3) == 1 && cache.stride(1) == 584 &&
             idx.numel() % batch == 0 && lens.numel() == batch);
        return {cache.data_ptr(), cache.stride(0), static_cast<const int32_t*>(idx.data_ptr()), static_cast<const int32_t*>(lens.data_ptr()),
                int32(cache.size(0)), int32(cache.size(1)), int32(idx.numel() / batch)};
    };
    const Pool swa = pool(p + 1), cmp = pool(p + 4);
    a.swa_pool = swa.data, a.swa_stride = swa.stride, a.swa_indices = swa.indices, a.swa_lengths = swa.lengths, a.swa_pages = swa.pages,
    a.swa_entries_per_block = swa.entries, a.swa_capacity = swa.capacity;
    a.cmp_pool = cmp.data, a.cmp_stride = cmp.stride, a.cmp_indices = cmp.indices, a.cmp_lengths = cmp.lengths, a.cmp_pages = cmp.pages,
    a.cmp_entries_per_block = cmp.entries, a.cmp_capacity = cmp.capacity;
    if (p[7] != Py_None) {
        const Tensor& sink = dense(p[7], ScalarType::Float);
        need(sink.numel() == heads);
        a.attn_sink = static_cast<const float*>(sink.data_ptr());
    }
    void* stream = current_stream();
    const int64_t wanted = truth(p[11]) ? entries.wuda_sparse_mla_workspace_bytes(a.batch, a.heads, int32(int64_t(a.swa_capacity) + a.cmp_capacity)) : 0;
    need(wanted >= 0);
    std::optional<Scratch> scratch;
    if (wanted > 0) {
        scratch.emplace(p[12], q, stream, wanted);
        a.workspace = scratch->at, a.workspace_bytes = wanted;
    }
    Tensor made;
    if (p[9] == Py_None) made = at::empty_like(q);
    const Tensor& out = made.defined() ? made : dense(p[9], ScalarType::BFloat16);
    need(out.is_contiguous() && out.sizes() == q.sizes());
    a.out = out.data_ptr();
    call(entries.wuda_sparse_mla_decode, static_cast<const wuda_sparse_mla_args*>(&a), status_of(p[10]), stream);
    return result(p[9], made);
}

// ---------------------------------------------------------------- module
template <PyObject* (*F)(PyObject* const*), Py_ssize_t N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != N) {
        PyErr_Format(PyExc_TypeError, "%d arguments are expected (got %d)", static_cast<int>(N), static_cast<int>(n));
        return nullptr;
    }
    try {
        need_plain_mode();
        return F(args);
    } catch (...) {      // also what torch throws for a tensor without storage and the like: the Python function says it again
    }
    if (PyErr_Occurred()) PyErr_Clear();
    Py_RETURN_NONE;
}

// The handle of the loaded library (ctypes.CDLL._handle).
PyObject* bind(PyObject*, PyObject* handle) {
    void* lib = PyLong_AsVoidPtr(handle);
    if (PyErr_Occurred()) return nullptr;
#define X(name)                                                                            \
    entries.name = reinterpret_cast<decltype(&::name)>(dlsym(lib, #name));                 \
    if (!entries.name) return PyErr_Format(PyExc_ImportError, "the library lacks " #name);
    WUDA_ENTRIES(X)
#undef X
    Py_RETURN_NONE;
}

#define WUDA_METHOD(name, f, n) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<f, n>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr},
                         WUDA_METHOD("mqa_logits_fp8", mqa_logits_fp8, 10),
                         WUDA_METHOD("mqa_logits_fp4", mqa_logits_fp4, 11),
                         WUDA_METHOD("topk", topk, 7),
                         WUDA_METHOD("rmsnorm_quant", rmsnorm_quant, 6),
                         WUDA_METHOD("act_quant", act_quant, 2),
                         WUDA_METHOD("rope_quant", rope_quant, 9),
                         WUDA_METHOD("fp8_gemm", fp8_gemm, 8),
                         WUDA_METHOD("fp4_gemm", fp4_gemm, 7),
                         WUDA_METHOD("bf16_gemm", bf16_gemm, 6),
                         WUDA_METHOD("nvfp4_gemm", nvfp4_gemm, 9),
                         WUDA_METHOD("sparse_mla_decode", sparse_mla_decode, 13),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fast() { return PyModule_Create(&module); }
