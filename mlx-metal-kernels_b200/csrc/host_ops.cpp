// Native call path of the operators (extension module lib/_b200q_host.so).
//
// An operator call on the ordinary arguments - CUDA tensors on the current device, contiguous, the dtypes and shapes the
// kernels read as they are - is checked, given its outputs and launched here, in a few microseconds of host time.  Every
// other call (a shape that does not match, a dtype to convert, a CPU tensor, a refused backend, an error code) makes the
// function return None, and the Python body of the operator takes it from the start: it holds all conversions and all
// error messages.  Nothing is kept between calls; outputs and scratch come from torch's caching allocator, which orders
// their reuse by stream.
//
// Why native: the Python route (validation, data_ptr() and ctypes conversions, current_stream()) costs about 17 us for a
// matvec whose kernel takes 5 us, and 25 us for an attention call of 13 us (host time per call, one B200 box).
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace {

using at::Tensor;

// addresses of the C ABI functions, handed over by the ctypes loader (the library itself is loaded there)
int (*p_qmatvec)(int, const void*, const uint8_t*, const void*, const void*, const void*, void*, int, int64_t, int64_t, int, int,
                 int, void*) = nullptr;
int (*p_gate_up)(int, const void*, const uint8_t*, const uint8_t*, const void*, const void*, const void*, const void*, void*, void*,
                 void*, const void*, const void*, int, float, void*, void*, int, int64_t, int64_t, int, int, int, void*) = nullptr;
int (*p_scratch_next)(void*, size_t) = nullptr;
size_t (*p_scratch_bytes)(int, int64_t, int) = nullptr;
size_t (*p_attn_ws)(int, int, int, int) = nullptr;
int (*p_attn_launches)(int, int, int) = nullptr;
int (*p_attn)(int, const void*, const uint8_t*, const uint8_t*, const void*, const void*, const int32_t*, const int32_t*, void*,
              void*, size_t, int, int, int, int, int, int64_t, int, int, float, int, int, void*) = nullptr;
int (*p_attn_window)(int, const void*, const uint8_t*, const uint8_t*, const void*, const void*, const int32_t*, const int32_t*,
                     void*, void*, size_t, int, int, int, int, int, int64_t, int, int, float, int, int, int, int, void*) = nullptr;

size_t (*p_plain_ws)(int, int, int, int) = nullptr;
int (*p_plain_attn)(const void*, const void*, const void*, const int32_t*, const int32_t*, void*, void*, size_t, int, int, int, int, int,
                    int64_t, int, float, int, void*) = nullptr;
int (*p_plain_checked)(const void*, const void*, const void*, const int32_t*, const int32_t*, void*, void*, size_t, int, int, int, int, int,
                       int64_t, int, float, int, int32_t*, void*) = nullptr;
int (*p_quant_pair)(int, const void*, const void*, uint8_t*, uint8_t*, void*, void*, int64_t, int, int, int, void*) = nullptr;
int (*p_dequant_pair)(int, const uint8_t*, const uint8_t*, const void*, const void*, void*, void*, int64_t, int, int, void*) = nullptr;

constexpr int kMaxDevices = 64;
constexpr int kErrUnsupported = -2, kErrWorkspace = -4;      // B200Q_ERR_*
constexpr int kMinNormRows = 5;      // from this many rows on the library runs the rmsnorm as a launch of its own

PyObject* none() { Py_RETURN_NONE; }

const Tensor* as_tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

bool safe_mode() {
    const char* v = std::getenv("MLX_METAL_CI_SAFE_MODE");
    return v != nullptr && std::strcmp(v, "1") == 0;
}

int dtype_code(at::ScalarType t) {
    return t == at::kHalf ? 0 : t == at::kBFloat16 ? 1 : t == at::kFloat ? 2 : -1;
}
bool act_dtype(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }

bool on(const Tensor& t, int dev) { return t.is_cuda() && t.get_device() == dev && t.is_contiguous(); }
bool is_matrix(const Tensor& t, int64_t r, int64_t c) { return t.dim() == 2 && t.size(0) == r && t.size(1) == c; }

// codes [n, row bytes of k], scales and zero points [n, groups] in one dtype
struct Matrix {
    const Tensor *w, *s, *z;
    int64_t n;
};
bool matrix(Matrix& m, PyObject* w, PyObject* s, PyObject* z, int bits, int64_t k, int64_t group, int dev) {
    m.w = as_tensor(w);
    m.s = as_tensor(s);
    m.z = z == Py_None ? nullptr : as_tensor(z);
    if (m.w == nullptr || m.s == nullptr || (m.z == nullptr && z != Py_None)) return false;
    if (m.w->dim() != 2 || m.w->scalar_type() != at::kByte || !on(*m.w, dev)) return false;
    m.n = m.w->size(0);
    if (m.n <= 0 || m.w->size(1) * (bits == 4 ? 2 : 1) != k) return false;
    const int64_t groups = (k + group - 1) / group;
    if (dtype_code(m.s->scalar_type()) < 0 || !on(*m.s, dev) || !is_matrix(*m.s, m.n, groups)) return false;
    return m.z == nullptr || (m.z->scalar_type() == m.s->scalar_type() && on(*m.z, dev) && is_matrix(*m.z, m.n, groups));
}
const void* ptr(const Tensor* t) { return t == nullptr ? nullptr : t->const_data_ptr(); }
const uint8_t* codes(const Tensor* t) { return static_cast<const uint8_t*>(t->const_data_ptr()); }

Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, int dev) {
    return at::detail::empty_cuda(shape, dtype, at::Device(at::kCUDA, dev), std::nullopt);
}
void* stream_of(int dev) { return c10::cuda::getCurrentCUDAStream(dev).stream(); }
// the device of the first tensor when it is the current one (the library launches on the current device), else -1
int current_device_of(const Tensor* t) {
    if (t == nullptr || !t->is_cuda()) return -1;
    const int dev = t->get_device();
    return dev == c10::cuda::current_device() ? dev : -1;
}
bool one_of(PyObject* s, std::initializer_list<const char*> names) {
    if (!PyUnicode_Check(s)) return false;
    for (const char* n : names)
        if (PyUnicode_CompareWithASCIIString(s, n) == 0) return true;
    return false;
}
// a plain int (not a bool or a float that Python's own arithmetic would treat differently)
bool as_int(PyObject* o, int64_t* v) {
    if (!PyLong_CheckExact(o)) return false;
    int overflow = 0;
    *v = PyLong_AsLongLongAndOverflow(o, &overflow);
    return overflow == 0;
}

// matvec(bits, x, w, scales, zeros, group_size, backend) -> y or None
PyObject* matvec(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    int64_t bits, group;
    if (p_qmatvec == nullptr || n_args != 7 || !as_int(a[0], &bits) || !as_int(a[5], &group) || group <= 0) return none();
    if (!one_of(a[6], {"cuda", "auto", "metal", "metal_tiled", "metal_parallel"}) || safe_mode()) return none();
    const Tensor* x = as_tensor(a[1]);
    const int dev = current_device_of(x);
    if (dev < 0 || !x->is_contiguous() || !act_dtype(x->scalar_type())) return none();
    if (!(x->dim() == 2 || (x->dim() == 3 && x->size(1) == 1))) return none();
    const int64_t B = x->size(0), K = x->size(x->dim() - 1);
    Matrix m;
    if (B <= 0 || B > INT32_MAX || K <= 0 || !matrix(m, a[2], a[3], a[4], (int)bits, K, group, dev)) return none();
    Tensor y = empty({B, m.n}, x->scalar_type(), dev), scratch;
    const size_t scratch_bytes = p_scratch_bytes((int)B, K, dtype_code(x->scalar_type()));
    if (scratch_bytes) scratch = empty({(int64_t)scratch_bytes}, at::kByte, dev);
    p_scratch_next(scratch_bytes ? scratch.mutable_data_ptr() : nullptr, scratch_bytes);      // the call below takes it, always
    const int rc = p_qmatvec((int)bits, x->const_data_ptr(), codes(m.w), ptr(m.s), ptr(m.z), nullptr, y.mutable_data_ptr(), (int)B, m.n,
                             K, (int)group, dtype_code(x->scalar_type()), dtype_code(m.s->scalar_type()), stream_of(dev));
    return rc == 0 ? THPVariable_Wrap(std::move(y)) : none();
}

// mlp_block(x, residual, norm_weight, gw, gs, gz, uw, us, uz, dw, ds, dz, bits, group_size, eps) -> out or None
PyObject* mlp_block(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    int64_t bits, group;
    if (p_gate_up == nullptr || n_args != 15 || !as_int(a[12], &bits) || !as_int(a[13], &group) || group <= 0 ||
        (bits != 4 && bits != 8) || !PyFloat_Check(a[14]) || safe_mode())
        return none();
    const Tensor *x = as_tensor(a[0]), *res = as_tensor(a[1]), *nw = as_tensor(a[2]);
    const int dev = current_device_of(x);
    if (dev < 0 || res == nullptr || nw == nullptr || x->dim() != 3 || x->sizes() != res->sizes() || !x->is_contiguous() ||
        !on(*res, dev) || !on(*nw, dev) || !act_dtype(x->scalar_type()) || res->scalar_type() != x->scalar_type() ||
        dtype_code(nw->scalar_type()) < 0)
        return none();
    const int64_t D = x->size(2), rows = x->size(0) * x->size(1);
    if (rows <= 0 || rows > INT32_MAX || nw->dim() != 1 || nw->size(0) != D) return none();
    Matrix g, u, d;
    if (!matrix(g, a[3], a[4], a[5], (int)bits, D, group, dev) || !matrix(u, a[6], a[7], a[8], (int)bits, D, group, dev) || u.n != g.n ||
        !matrix(d, a[9], a[10], a[11], (int)bits, g.n, group, dev) || d.n != D || u.s->scalar_type() != g.s->scalar_type() ||
        (u.z != nullptr && u.z->scalar_type() != g.s->scalar_type()))
        return none();
    const int act = dtype_code(x->scalar_type());
    void* st = stream_of(dev);
    // one scratch block: z [rows, D], the SwiGLU rows [rows, inter], and the normalised rows where the library wants them
    const int64_t zb = (rows * D * 2 + 255) / 256 * 256, mb = (rows * g.n * 2 + 255) / 256 * 256;
    const bool want_normed = rows >= kMinNormRows;
    const size_t xb = std::max(p_scratch_bytes((int)rows, D, act), p_scratch_bytes((int)rows, g.n, act));
    Tensor scratch = empty({zb + mb + (want_normed ? zb : 0) + (int64_t)xb}, at::kByte, dev);
    uint8_t* z = static_cast<uint8_t*>(scratch.mutable_data_ptr());
    uint8_t *mlp = z + zb, *normed = want_normed ? mlp + mb : nullptr;
    Tensor out = empty(x->sizes(), x->scalar_type(), dev);
    void* xs = xb ? z + zb + mb + (want_normed ? zb : 0) : nullptr;
    const float eps = (float)PyFloat_AS_DOUBLE(a[14]);
    p_scratch_next(xs, xb);
    int rc = p_gate_up((int)bits, x->const_data_ptr(), codes(g.w), codes(u.w), ptr(g.s), ptr(u.s), ptr(g.z), ptr(u.z), nullptr, nullptr,
                       mlp, res->const_data_ptr(), nw->const_data_ptr(), dtype_code(nw->scalar_type()), eps, z, normed, (int)rows, g.n,
                       D, (int)group, act, dtype_code(g.s->scalar_type()), st);
    if (rc != 0) return none();
    p_scratch_next(xs, xb);
    rc = p_qmatvec((int)bits, mlp, codes(d.w), ptr(d.s), ptr(d.z), z, out.mutable_data_ptr(), (int)rows, D, g.n, (int)group, act,
                   dtype_code(d.s->scalar_type()), st);
    return rc == 0 ? THPVariable_Wrap(std::move(out)) : none();
}

PyObject *s_bits, *s_group_size, *s_shape, *s_kq, *s_vq, *s_ks, *s_vs, *s_bt, *s_len;

// Owned attribute, released at scope end.
struct Attr {
    PyObject* o;
    Attr(PyObject* obj, PyObject* name) : o(PyObject_GetAttr(obj, name)) {
        if (o == nullptr) PyErr_Clear();
    }
    ~Attr() { Py_XDECREF(o); }
    Attr(const Attr&) = delete;
};

// paged_attention(q, cache, scale or None, sink_tokens, window_size) -> out or None
PyObject* paged_attention(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    int64_t sink, window;
    if (p_attn == nullptr || n_args != 5 || !as_int(a[3], &sink) || !as_int(a[4], &window)) return none();
    const Tensor* q = as_tensor(a[0]);
    const int dev = current_device_of(q);
    if (dev < 0 || q->dim() != 4 || q->size(1) != 1 || !q->is_contiguous() || !act_dtype(q->scalar_type())) return none();
    const int64_t B = q->size(0), Hq = q->size(2), D = q->size(3);
    Attr bits_o(a[1], s_bits), group_o(a[1], s_group_size), shape(a[1], s_shape), kq_o(a[1], s_kq), vq_o(a[1], s_vq), ks_o(a[1], s_ks),
        vs_o(a[1], s_vs), bt_o(a[1], s_bt), len_o(a[1], s_len);
    int64_t bits, group, dims[4];
    if (bits_o.o == nullptr || group_o.o == nullptr || shape.o == nullptr || kq_o.o == nullptr || vq_o.o == nullptr ||
        ks_o.o == nullptr || vs_o.o == nullptr || bt_o.o == nullptr || len_o.o == nullptr)
        return none();
    if (!as_int(bits_o.o, &bits) || !as_int(group_o.o, &group) || (bits != 4 && bits != 8) || group <= 0 || !PyTuple_Check(shape.o) ||
        PyTuple_GET_SIZE(shape.o) != 4)
        return none();
    for (int i = 0; i < 4; ++i)
        if (!as_int(PyTuple_GET_ITEM(shape.o, i), &dims[i]) || dims[i] <= 0) return none();
    const int64_t pages = dims[0], P = dims[1], Hkv = dims[2];
    const Tensor *kq = as_tensor(kq_o.o), *vq = as_tensor(vq_o.o), *ks = as_tensor(ks_o.o), *vs = as_tensor(vs_o.o),
                 *bt = as_tensor(bt_o.o), *len = as_tensor(len_o.o);
    if (!kq || !vq || !ks || !vs || !bt || !len || !on(*kq, dev) || !on(*vq, dev) || !on(*ks, dev) || !on(*vs, dev) || !on(*bt, dev) ||
        !on(*len, dev))
        return none();
    const int64_t slots = pages * P * Hkv, dp = bits == 4 ? (D + 1) / 2 : D, gd = (D + group - 1) / group;
    if (B <= 0 || Hq <= 0 || D <= 0 || D > 128 || D != dims[3] || Hq < Hkv || Hq % Hkv != 0 || kq->scalar_type() != at::kByte ||
        vq->scalar_type() != at::kByte || kq->numel() != slots * dp || vq->numel() != slots * dp || ks->numel() != slots * gd ||
        vs->numel() != slots * gd || dtype_code(ks->scalar_type()) < 0 || vs->scalar_type() != ks->scalar_type() ||
        bt->scalar_type() != at::kInt || bt->dim() != 2 || bt->size(0) != B || len->scalar_type() != at::kInt || len->numel() != B ||
        B > INT32_MAX || Hq > INT32_MAX || P > INT32_MAX || bt->size(1) > INT32_MAX || bt->size(1) <= 0)
        return none();
    double scale = 1.0 / std::sqrt((double)D);
    if (a[2] != Py_None) {
        if (!PyFloat_Check(a[2])) return none();
        scale = PyFloat_AS_DOUBLE(a[2]);
    }
    Tensor out = empty(q->sizes(), q->scalar_type(), dev);
    // scratch for split-KV partial results; the one-launch cluster kernel of small dense batches needs none
    Tensor ws;
    size_t ws_bytes = 0;
    if (window > 0 || p_attn_launches((int)B, (int)Hkv, 0) > 1) {
        ws_bytes = p_attn_ws((int)B, (int)Hq, (int)Hkv, (int)D);
        ws = empty({(int64_t)ws_bytes}, at::kByte, dev);
    }
    const auto i32 = [](const Tensor* t) { return static_cast<const int32_t*>(t->const_data_ptr()); };
    void* wp = ws_bytes ? ws.mutable_data_ptr() : nullptr;
    const int act = dtype_code(q->scalar_type()), sdt = dtype_code(ks->scalar_type()), mb = (int)bt->size(1);
    const int rc = window > 0
        ? p_attn_window((int)bits, q->const_data_ptr(), codes(kq), codes(vq), ptr(ks), ptr(vs), i32(bt), i32(len), out.mutable_data_ptr(), wp,
                        ws_bytes, (int)B, (int)Hq, (int)Hkv, (int)D, (int)P, pages, mb, (int)group, (float)scale, act, sdt, (int)sink,
                        (int)window, stream_of(dev))
        : p_attn((int)bits, q->const_data_ptr(), codes(kq), codes(vq), ptr(ks), ptr(vs), i32(bt), i32(len), out.mutable_data_ptr(), wp,
                 ws_bytes, (int)B, (int)Hq, (int)Hkv, (int)D, (int)P, pages, mb, (int)group, (float)scale, act, sdt, stream_of(dev));
    return rc == 0 ? THPVariable_Wrap(std::move(out)) : none();
}

// Queries and waits on a stream are refused to every thread while one captures a graph in the default mode, unless the thread asks
// for the relaxed one.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
// Memory that a kernel on the stream may still write to goes back to its allocator when the stream has ended; if even the wait
// fails it is kept for good.
void release_after_stream(Tensor word, cudaStream_t st) {
    cudaError_t err;
    Py_BEGIN_ALLOW_THREADS
    const RelaxedCapture relaxed;
    err = cudaStreamSynchronize(st);
    Py_END_ALLOW_THREADS
    if (err != cudaSuccess) new Tensor(std::move(word));
}

// plain_attention(q, K, V, block_table, lengths, scale or None) -> out or None: fp16 / bf16 pages.  The lengths are
// range-checked on the host, as the operator promises.  The split-KV kernel reports on them at its start, into pinned memory that
// the host polls while the GPU goes on (a copy on the stream took 10 of 42 us per call at 16 sequences: it kept the kernel from
// starting under the one before).  Elsewhere they are copied out ahead of the kernels, which clamp what they read,
// and the host waits for that copy once the kernels are enqueued.
PyObject* plain_attention(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    if (p_plain_attn == nullptr || n_args != 6 || safe_mode()) return none();
    const Tensor *q = as_tensor(a[0]), *k = as_tensor(a[1]), *v = as_tensor(a[2]), *bt = as_tensor(a[3]), *len = as_tensor(a[4]);
    const int dev = current_device_of(q);
    if (dev < 0 || dev >= kMaxDevices || !k || !v || !bt || !len || q->dim() != 4 || q->size(1) != 1 || !q->is_contiguous() ||
        !act_dtype(q->scalar_type()))
        return none();
    const int64_t B = q->size(0), Hq = q->size(2), D = q->size(3);
    if (!on(*k, dev) || !on(*v, dev) || !on(*bt, dev) || !on(*len, dev) || k->dim() != 4 || k->sizes() != v->sizes() ||
        k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || k->size(3) != D || bt->dim() != 2 ||
        bt->size(0) != B || bt->scalar_type() != at::kInt || len->scalar_type() != at::kInt || len->dim() != 1 || len->size(0) != B)
        return none();
    const int64_t pages = k->size(0), P = k->size(1), Hkv = k->size(2), mb = bt->size(1);
    if (B <= 0 || Hq <= 0 || D <= 0 || D > 128 || pages <= 0 || P <= 0 || Hkv <= 0 || mb <= 0 || Hq % Hkv != 0 || B > INT32_MAX ||
        Hq > INT32_MAX || P * mb > INT32_MAX)
        return none();
    double scale = 1.0 / std::sqrt((double)D);
    if (a[5] != Py_None) {
        if (!PyFloat_Check(a[5])) return none();
        scale = PyFloat_AS_DOUBLE(a[5]);
    }
    cudaStream_t st = (cudaStream_t)stream_of(dev);
    cudaStreamCaptureStatus capture;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) return none();
    Tensor out = empty(q->sizes(), q->scalar_type(), dev);
    const size_t ws_bytes = p_plain_ws((int)B, (int)Hq, (int)Hkv, (int)mb);
    Tensor ws = empty({(int64_t)std::max<size_t>(ws_bytes, 16)}, at::kByte, dev);
    if (D == 128 && P == 16) {
        Tensor word = at::detail::empty_cpu({1}, at::kInt, std::nullopt, std::nullopt, /*pin_memory=*/true, std::nullopt);
        volatile int32_t* verdict = static_cast<volatile int32_t*>(word.mutable_data_ptr());
        *verdict = 0;
        const int rc = p_plain_checked(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), static_cast<const int32_t*>(bt->const_data_ptr()),
                                       static_cast<const int32_t*>(len->const_data_ptr()), out.mutable_data_ptr(), ws.mutable_data_ptr(), ws_bytes,
                                       (int)B, (int)Hq, (int)Hkv, (int)D, (int)P, pages, (int)mb, (float)scale, dtype_code(q->scalar_type()),
                                       const_cast<int32_t*>(verdict), st);
        if (rc == 0) {
            Py_BEGIN_ALLOW_THREADS
            // the stream is asked now and then, so that a kernel that never ran (an earlier error) ends the wait
            const RelaxedCapture relaxed;
            for (uint32_t i = 1; *verdict == 0; ++i) {
                if (i % 4096 == 0 && cudaStreamQuery(st) != cudaErrorNotReady) break;
                __builtin_ia32_pause();
            }
            Py_END_ALLOW_THREADS
            if (*verdict == 0) release_after_stream(word, st);
            return *verdict == 1 ? THPVariable_Wrap(std::move(out)) : none();      // 2: the Python body raises
        }
        if (rc != kErrUnsupported && rc != kErrWorkspace) {      // nothing is launched with these two; else the main kernel may be
            release_after_stream(word, st);
            return none();
        }
    }
    static thread_local cudaEvent_t copied[kMaxDevices] = {};      // one per thread and device that ever calls this
    if (copied[dev] == nullptr && cudaEventCreateWithFlags(&copied[dev], cudaEventDisableTiming) != cudaSuccess) return none();
    Tensor host = at::detail::empty_cpu({B}, at::kInt, std::nullopt, std::nullopt, /*pin_memory=*/true, std::nullopt);
    if (cudaMemcpyAsync(host.mutable_data_ptr(), len->const_data_ptr(), (size_t)B * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaEventRecord(copied[dev], st) != cudaSuccess) {
        release_after_stream(host, st);
        return none();
    }
    const int rc = p_plain_attn(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), static_cast<const int32_t*>(bt->const_data_ptr()),
                                static_cast<const int32_t*>(len->const_data_ptr()), out.mutable_data_ptr(), ws.mutable_data_ptr(), ws_bytes,
                                (int)B, (int)Hq, (int)Hkv, (int)D, (int)P, pages, (int)mb, (float)scale, dtype_code(q->scalar_type()), st);
    cudaError_t err;
    Py_BEGIN_ALLOW_THREADS
    const RelaxedCapture relaxed;
    err = cudaEventSynchronize(copied[dev]);
    Py_END_ALLOW_THREADS
    if (err != cudaSuccess) release_after_stream(host, st);
    if (rc != 0 || err != cudaSuccess) return none();
    const int32_t* n = static_cast<const int32_t*>(host.const_data_ptr());
    for (int64_t b = 0; b < B; ++b)
        if (n[b] < 0 || n[b] > mb * P) return none();              // the Python body raises
    return THPVariable_Wrap(std::move(out));
}

PyObject* tuple_of(std::initializer_list<Tensor*> ts) {
    PyObject* out = PyTuple_New((Py_ssize_t)ts.size());
    Py_ssize_t i = 0;
    for (Tensor* t : ts) PyTuple_SET_ITEM(out, i++, THPVariable_Wrap(std::move(*t)));
    return out;
}

// quantize_kv(K, V, bits, group_size) -> (k codes, v codes, k scales, v scales) or None; K, V [..., D] of one shape
PyObject* quantize_kv(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    int64_t bits, group;
    if (p_quant_pair == nullptr || n_args != 4 || !as_int(a[2], &bits) || !as_int(a[3], &group) || (bits != 4 && bits != 8) || group <= 0)
        return none();
    const Tensor *k = as_tensor(a[0]), *v = as_tensor(a[1]);
    const int dev = current_device_of(k);
    if (dev < 0 || v == nullptr || k->dim() < 1 || k->sizes() != v->sizes() || !on(*k, dev) || !on(*v, dev) || !act_dtype(k->scalar_type()) ||
        v->scalar_type() != k->scalar_type() || k->numel() == 0)
        return none();
    const int64_t D = k->size(-1);
    if (D > INT32_MAX || group > INT32_MAX) return none();
    std::vector<int64_t> shape(k->sizes().begin(), k->sizes().end());
    shape.back() = bits == 4 ? (D + 1) / 2 : D;
    Tensor kc = empty(shape, at::kByte, dev), vc = empty(shape, at::kByte, dev);
    shape.back() = (D + group - 1) / group;
    Tensor ks = empty(shape, at::kHalf, dev), vs = empty(shape, at::kHalf, dev);
    const auto u8 = [](Tensor& t) { return static_cast<uint8_t*>(t.mutable_data_ptr()); };
    const int rc = p_quant_pair((int)bits, k->const_data_ptr(), v->const_data_ptr(), u8(kc), u8(vc), ks.mutable_data_ptr(),
                                vs.mutable_data_ptr(), k->numel() / D, (int)D, (int)group, dtype_code(k->scalar_type()), stream_of(dev));
    return rc == 0 ? tuple_of({&kc, &vc, &ks, &vs}) : none();
}

// dequantize_kv(k codes, v codes, k scales, v scales, bits, group_size, shape) -> (K, V) fp16 of `shape`, or None
PyObject* dequantize_kv(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    int64_t bits, group;
    if (p_dequant_pair == nullptr || n_args != 7 || !as_int(a[4], &bits) || !as_int(a[5], &group) || (bits != 4 && bits != 8) ||
        group <= 0 || !PyTuple_Check(a[6]))
        return none();
    const Tensor *kc = as_tensor(a[0]), *vc = as_tensor(a[1]), *ks = as_tensor(a[2]), *vs = as_tensor(a[3]);
    const int dev = current_device_of(kc);
    if (dev < 0 || !vc || !ks || !vs || !on(*kc, dev) || !on(*vc, dev) || !on(*ks, dev) || !on(*vs, dev) || kc->scalar_type() != at::kByte ||
        vc->scalar_type() != at::kByte || ks->scalar_type() != at::kHalf || vs->scalar_type() != at::kHalf)
        return none();
    std::vector<int64_t> shape((size_t)PyTuple_GET_SIZE(a[6]));
    int64_t n = 1;
    for (size_t i = 0; i < shape.size(); ++i) {
        if (!as_int(PyTuple_GET_ITEM(a[6], i), &shape[i]) || shape[i] <= 0) return none();
        n *= shape[i];
    }
    if (shape.empty() || shape.back() > INT32_MAX || group > INT32_MAX) return none();
    const int64_t D = shape.back(), rows = n / D, dp = bits == 4 ? (D + 1) / 2 : D, gd = (D + group - 1) / group;
    if (kc->numel() != rows * dp || vc->numel() != rows * dp || ks->numel() != rows * gd || vs->numel() != rows * gd) return none();
    Tensor k = empty(shape, at::kHalf, dev), v = empty(shape, at::kHalf, dev);
    const int rc = p_dequant_pair((int)bits, codes(kc), codes(vc), ptr(ks), ptr(vs), k.mutable_data_ptr(), v.mutable_data_ptr(), rows, (int)D,
                                  (int)group, stream_of(dev));
    return rc == 0 ? tuple_of({&k, &v}) : none();
}

// bind({symbol: address}): the C ABI functions to call
PyObject* bind(PyObject*, PyObject* table) {
    const struct { const char* name; void** slot; } want[] = {
        {"b200q_qmatvec", (void**)&p_qmatvec}, {"b200q_gate_up_swiglu", (void**)&p_gate_up},
        {"b200q_scratch_next", (void**)&p_scratch_next}, {"b200q_scratch_bytes", (void**)&p_scratch_bytes},
        {"b200q_paged_gqa_workspace_bytes", (void**)&p_attn_ws}, {"b200q_attention_stage_launches", (void**)&p_attn_launches},
        {"b200q_paged_gqa_decode", (void**)&p_attn}, {"b200q_paged_gqa_decode_window", (void**)&p_attn_window},
        {"b200q_paged_fp16_gqa_workspace_bytes", (void**)&p_plain_ws}, {"b200q_paged_fp16_gqa_decode", (void**)&p_plain_attn},
        {"b200q_paged_fp16_gqa_decode_checked", (void**)&p_plain_checked},
        {"b200q_quantize_kv_pair", (void**)&p_quant_pair}, {"b200q_dequantize_kv_pair", (void**)&p_dequant_pair},
    };
    for (const auto& w : want) {
        PyObject* v = PyDict_GetItemString(table, w.name);
        void* p = v == nullptr ? nullptr : PyLong_AsVoidPtr(v);
        if (p == nullptr) {
            PyErr_Format(PyExc_KeyError, "%s", w.name);
            return nullptr;
        }
        *w.slot = p;
    }
    return none();
}

// C++ exceptions (out of memory, a CUDA error) become Python ones, as torch's own functions raise them
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    return F(self, args, n);
    END_HANDLE_TH_ERRORS
}
#define FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<fn>))

PyMethodDef methods[] = {
    {"bind", bind, METH_O, "bind({symbol: address})"},
    {"matvec", FAST(matvec), METH_FASTCALL, nullptr},
    {"mlp_block", FAST(mlp_block), METH_FASTCALL, nullptr},
    {"quantize_kv", FAST(quantize_kv), METH_FASTCALL, nullptr},
    {"dequantize_kv", FAST(dequantize_kv), METH_FASTCALL, nullptr},
    {"plain_attention", FAST(plain_attention), METH_FASTCALL, nullptr},
    {"paged_attention", FAST(paged_attention), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_b200q_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__b200q_host() {
    const struct { const char* name; PyObject** slot; } names[] = {
        {"bits", &s_bits}, {"group_size", &s_group_size}, {"original_page_shape", &s_shape},
        {"k_pages_q", &s_kq}, {"v_pages_q", &s_vq}, {"k_scales", &s_ks}, {"v_scales", &s_vs}, {"block_table", &s_bt}, {"lengths", &s_len},
    };
    for (const auto& n : names)
        if ((*n.slot = PyUnicode_InternFromString(n.name)) == nullptr) return nullptr;
    return PyModule_Create(&module_def);
}
