// Python operators over the C ABI (module nacho_b200._native). A call on small operands computes for a few
// microseconds, so what surrounds it counts: this module reads the tensors of the operand objects, takes the
// result arrays from torch's caching allocator, runs one C-ABI entry point without the interpreter lock and
// hands back an object of the caller's class -- about 4 us where the same steps in Python with ctypes took
// 35. It computes nothing itself. Classes, slots and error texts are those of nacho/nacho_ext.py, which
// hands them over with bind().
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <exception>
#include <map>
#include <mutex>
#include <utility>

#include "nacho_b200.h"

namespace {

// ---- what nacho_ext.py binds ---------------------------------------------------------------

enum Kind { CSR = 0, COO = 1, DCSR = 2, COO3 = 3, CSF3 = 4, SCALAR = 5, KINDS = 6 };
PyTypeObject *g_class[KINDS] = {};
PyObject *g_check = nullptr;  // check(status, where): raises on a non-zero status
PyObject *g_name[9] = {};    // interned slot names
enum Name { N_offsets, N_indices, N_values, N_dims, N_i, N_j, N_k, N_jp, N_kp, NAMES };
const char *const NAME_TEXT[NAMES] = {"_offsets", "_indices", "_values", "_dims", "_i", "_j", "_k", "_jp", "_kp"};

struct PyFailure {};  // a Python exception is set

struct Ref {  // owned reference
    PyObject *p;
    explicit Ref(PyObject *o) : p(o) { if (!o) throw PyFailure(); }
    ~Ref() { Py_XDECREF(p); }
    Ref(const Ref &) = delete;
    PyObject *release() { PyObject *r = p; p = nullptr; return r; }
};

const at::Tensor &tensor_of(PyObject *obj, Name slot) {
    Ref t(PyObject_GetAttr(obj, g_name[slot]));
    if (!THPVariable_Check(t.p)) {
        PyErr_SetString(PyExc_TypeError, "operand slot does not hold a tensor");
        throw PyFailure();
    }
    return THPVariable_Unpack(t.p);  // the operand object keeps it alive while the interpreter lock is held
}

template <int N>
void dims_of(PyObject *obj, int32_t *out) {
    Ref d(PyObject_GetAttr(obj, g_name[N_dims]));
    if (!PyTuple_Check(d.p) || PyTuple_GET_SIZE(d.p) != N) {
        PyErr_SetString(PyExc_TypeError, "operand has no extents");
        throw PyFailure();
    }
    for (int k = 0; k < N; ++k) out[k] = (int32_t)PyLong_AsLong(PyTuple_GET_ITEM(d.p, k));
}

void need_kind(PyObject *obj, Kind kind, const char *where, const char *what) {
    if (Py_TYPE(obj) == g_class[kind]) return;
    const int is = PyObject_IsInstance(obj, reinterpret_cast<PyObject *>(g_class[kind]));
    if (is < 0) throw PyFailure();
    if (!is) {
        PyErr_Format(PyExc_TypeError, "%s: operands must be %s", where, what);
        throw PyFailure();
    }
}

// ---- operand views -------------------------------------------------------------------------

int32_t *ints(const at::Tensor &t) { return static_cast<int32_t *>(t.data_ptr()); }
float *floats(const at::Tensor &t) { return static_cast<float *>(t.data_ptr()); }

struct View {  // device and arrays of one operand, for what all kinds share
    c10::Device device = c10::Device(c10::kCPU);
    at::Tensor arrays[6];  // references of their own: another thread may give the operand new arrays meanwhile
    int n = 0;

    const at::Tensor &array(PyObject *o, Name slot) {
        arrays[n] = tensor_of(o, slot);
        return arrays[n++];
    }
    int32_t *index(PyObject *o, Name slot) { return ints(array(o, slot)); }
};

nb200_csr view_csr(PyObject *o, View &v) {
    const at::Tensor &val = v.array(o, N_values);
    int32_t d[2];
    dims_of<2>(o, d);
    v.device = val.device();
    return nb200_csr{d[0], d[1], (int32_t)val.numel(), v.index(o, N_offsets), v.index(o, N_indices), floats(val)};
}

nb200_coo view_coo(PyObject *o, View &v) {
    const at::Tensor &val = v.array(o, N_values);
    int32_t d[2];
    dims_of<2>(o, d);
    v.device = val.device();
    return nb200_coo{d[0], d[1], (int32_t)val.numel(), v.index(o, N_i), v.index(o, N_j), floats(val)};
}

nb200_dcsr view_dcsr(PyObject *o, View &v) {
    const at::Tensor &val = v.array(o, N_values), &i = v.array(o, N_i);
    int32_t d[2];
    dims_of<2>(o, d);
    v.device = val.device();
    return nb200_dcsr{d[0], d[1], (int32_t)i.numel(), (int32_t)val.numel(), ints(i), v.index(o, N_jp), v.index(o, N_j), floats(val)};
}

nb200_coo3 view_coo3(PyObject *o, View &v) {
    const at::Tensor &val = v.array(o, N_values);
    nb200_coo3 s{};
    dims_of<3>(o, s.dims);
    v.device = val.device();
    s.nnz = (int32_t)val.numel();
    s.i = v.index(o, N_i), s.j = v.index(o, N_j), s.k = v.index(o, N_k), s.val = floats(val);
    return s;
}

nb200_csf3 view_csf3(PyObject *o, View &v) {
    const at::Tensor &val = v.array(o, N_values), &i = v.array(o, N_i), &j = v.array(o, N_j), &k = v.array(o, N_k);
    nb200_csf3 s{};
    dims_of<3>(o, s.dims);
    v.device = val.device();
    s.n_i = (int32_t)i.numel(), s.n_j = (int32_t)j.numel(), s.n_k = (int32_t)k.numel();
    s.i_idx = ints(i), s.j_ptr = v.index(o, N_jp), s.j_idx = ints(j), s.k_ptr = v.index(o, N_kp), s.k_idx = ints(k), s.val = floats(val);
    return s;
}

void same_device(const View &a, const View &b) {
    if (a.device != b.device) {
        PyErr_SetString(PyExc_ValueError, "operands live on different devices");
        throw PyFailure();
    }
}

// ---- results -------------------------------------------------------------------------------

at::Tensor array(int64_t n, at::ScalarType type, c10::Device dev) {
    return at::Tensor(at::detail::empty_cuda({std::max<int64_t>(n, 1)}, type, dev, std::nullopt));
}
at::Tensor int_array(int64_t n, c10::Device dev) { return array(n, at::kInt, dev); }
at::Tensor float_array(int64_t n, c10::Device dev) { return array(n, at::kFloat, dev); }

// A result array was taken at its worst-case length; its tensor covers the part in use.
void used(at::Tensor &t, int64_t n) {
    t.unsafeGetTensorImpl()->set_sizes_contiguous(c10::IntArrayRef(&n, 1));
}

struct Result {
    Ref obj;
    explicit Result(Kind kind) : obj(g_class[kind]->tp_alloc(g_class[kind], 0)) {}
    void set(Name slot, at::Tensor &t) {
        Ref v(THPVariable_Wrap(t));
        if (PyObject_SetAttr(obj.p, g_name[slot], v.p) < 0) throw PyFailure();
    }
    template <int N>
    void dims(const int32_t *d) {
        Ref t(PyTuple_New(N));
        for (int k = 0; k < N; ++k) PyTuple_SET_ITEM(t.p, k, PyLong_FromLong(d[k]));
        if (PyObject_SetAttr(obj.p, g_name[N_dims], t.p) < 0) throw PyFailure();
    }
};

void check(int status, const char *where) {
    if (status == NB200_OK) return;
    Ref r(PyObject_CallFunction(g_check, "is", status, where));
    PyErr_Format(PyExc_RuntimeError, "%s: status %d", where, status);  // only if check() did not raise
    throw PyFailure();
}

struct NoLock {  // releases the interpreter lock
    PyThreadState *state = PyEval_SaveThread();
    ~NoLock() { PyEval_RestoreThread(state); }
};

// Calls of several host threads on one stream take turns at issuing their kernels: they share the stream's scratch
// arrays and result words. The lock's key is the pool's, device and stream: the default stream has the same handle
// on every device, and a lock is held while its call waits for a length. (Locks stay, as the pool's entries do.)
std::mutex &stream_lock(int device, void *stream) {
    static std::mutex guard;
    static std::map<std::pair<int, void *>, std::mutex> locks;
    thread_local std::pair<int, void *> last{-1, nullptr};
    thread_local std::mutex *last_lock = nullptr;
    const std::pair<int, void *> key{device, stream};
    if (!last_lock || last != key) {
        std::lock_guard<std::mutex> g(guard);
        last_lock = &locks[key];
        last = key;
    }
    return *last_lock;
}

// Runs a C-ABI call on the operands' device and the current stream of the caller, without the interpreter lock. A call
// returns when the result's length is known, with kernels still running: the allocator is told that the
// operands' arrays are in use on this stream, which matters when they came from another one.
template <size_t N, typename F>
int run(const View *const (&operands)[N], F call) {
    const c10::Device device = operands[0]->device;
    c10::cuda::CUDAGuard guard(device);
    const c10::cuda::CUDAStream current = c10::cuda::getCurrentCUDAStream(device.index());
    void *stream = current.stream();
    int status;
    {
        NoLock unlocked;
        std::lock_guard<std::mutex> turn(stream_lock(device.index(), stream));
        status = call(stream);
    }
    for (const View *operand : operands)
        for (int k = 0; k < operand->n; ++k) c10::cuda::CUDACachingAllocator::recordStream(operand->arrays[k].storage().data_ptr(), current);
    return status;
}

template <size_t N, typename F>
void launch(const View *const (&operands)[N], const char *where, F call) {
    check(run(operands, call), where);
}

// ---- operators -----------------------------------------------------------------------------

typedef int (*csr2_fn)(const nb200_csr *, const nb200_csr *, nb200_csr *, int64_t, void *);
typedef int (*coo2_fn)(const nb200_coo *, const nb200_coo *, nb200_coo *, int64_t, void *);
typedef int (*dcsr2_fn)(const nb200_dcsr *, const nb200_dcsr *, nb200_dcsr *, int64_t, int64_t, void *);

// A CSR result of up to `capacity` entries, filled by `call(z, stream)`.
template <size_t N, typename F>
PyObject *csr_result(const View *const (&operands)[N], const char *where, int32_t rows, int32_t cols, int64_t capacity, F call) {
    const c10::Device device = operands[0]->device;
    at::Tensor rp = int_array((int64_t)rows + 1, device), col = int_array(capacity, device), val = float_array(capacity, device);
    nb200_csr z{rows, cols, 0, ints(rp), ints(col), floats(val)};
    launch(operands, where, [&](void *stream) { return call(&z, stream); });
    used(col, z.nnz);
    used(val, z.nnz);
    Result r(CSR);
    r.set(N_offsets, rp), r.set(N_indices, col), r.set(N_values, val);
    const int32_t d[2] = {z.rows, z.cols};
    r.dims<2>(d);
    return r.obj.release();
}

PyObject *csr_binary(csr2_fn fn, bool is_union, const char *where, PyObject *const *args) {
    for (int k = 0; k < 2; ++k) need_kind(args[k], CSR, where, "CSR_gpu");
    View va, vb;
    const nb200_csr a = view_csr(args[0], va), b = view_csr(args[1], vb);
    same_device(va, vb);
    const int64_t capacity = is_union ? (int64_t)a.nnz + b.nnz : std::min(a.nnz, b.nnz);
    return csr_result({&va, &vb}, where, a.rows, a.cols, capacity, [&](nb200_csr *z, void *stream) { return fn(&a, &b, z, capacity, stream); });
}

PyObject *csr_add(PyObject *const *args) { return csr_binary(nb200_csr_add_f32_into, true, "gpu_csr_add_f32", args); }
PyObject *csr_mul(PyObject *const *args) { return csr_binary(nb200_csr_mul_f32_into, false, "gpu_csr_mul_f32", args); }

constexpr int64_t ADD3_POOL_BYTES = 8 << 20;

PyObject *csr_add_3(PyObject *const *args) {
    const char *where = "gpu_csr_add_3_f32";
    for (int k = 0; k < 3; ++k) need_kind(args[k], CSR, where, "CSR_gpu");
    View va, vb, vc;
    const nb200_csr a = view_csr(args[0], va), b = view_csr(args[1], vb), c = view_csr(args[2], vc);
    same_device(va, vb);
    same_device(va, vc);
    const int64_t capacity = (int64_t)a.nnz + b.nnz + c.nnz;
    // The intermediate sum is as large as the operands: it lies in an array of this call. Only a small one stays in the
    // library's pool (the array costs half a microsecond).
    const int64_t scratch_bytes = nb200_csr_add_3_f32_scratch(&a, &b, &c);
    if (scratch_bytes <= ADD3_POOL_BYTES)
        return csr_result({&va, &vb, &vc}, where, a.rows, a.cols, capacity,
                          [&](nb200_csr *z, void *stream) { return nb200_csr_add_3_f32_into(&a, &b, &c, z, capacity, stream); });
    at::Tensor scratch = array(scratch_bytes, at::kByte, va.device);
    return csr_result({&va, &vb, &vc}, where, a.rows, a.cols, capacity,
                      [&](nb200_csr *z, void *stream) { return nb200_csr_add_3_f32_lent(&a, &b, &c, z, capacity, scratch.data_ptr(), scratch_bytes, stream); });
}

PyObject *sssmm(PyObject *const *args) {
    const char *where = "gpu_sssmm_f32";
    for (int k = 0; k < 3; ++k) need_kind(args[k], CSR, where, "CSR_gpu");
    View va, vb, vc;
    const nb200_csr a = view_csr(args[0], va), b = view_csr(args[1], vb), c = view_csr(args[2], vc);
    same_device(va, vb);
    same_device(va, vc);
    return csr_result({&va, &vb, &vc}, where, a.rows, b.cols, c.nnz, [&](nb200_csr *z, void *stream) { return nb200_sssmm_f32_into(&a, &b, &c, z, c.nnz, stream); });
}

PyObject *coo_csr_add(PyObject *const *args) {
    const char *where = "gpu_coo_csr_add_f32";
    need_kind(args[0], CSR, where, "(CSR_gpu, COO_gpu)");
    need_kind(args[1], COO, where, "(CSR_gpu, COO_gpu)");
    View va, vb;
    const nb200_csr a = view_csr(args[0], va);
    const nb200_coo b = view_coo(args[1], vb);
    same_device(va, vb);
    const int64_t capacity = (int64_t)a.nnz + b.nnz;
    return csr_result({&va, &vb}, where, a.rows, a.cols, capacity, [&](nb200_csr *z, void *stream) { return nb200_coo_csr_add_f32_into(&a, &b, z, capacity, stream); });
}

PyObject *spgemm(PyObject *const *args) {
    const char *where = "gpu_spgemm_f32";
    for (int k = 0; k < 2; ++k) need_kind(args[k], CSR, where, "CSR_gpu");
    View va, vb;
    const nb200_csr a = view_csr(args[0], va), b = view_csr(args[1], vb);
    same_device(va, vb);
    at::Tensor rp = int_array((int64_t)a.rows + 1, va.device);
    nb200_csr c{a.rows, b.cols, 0, ints(rp), nullptr, nullptr};
    struct Taken {  // the result's arrays, taken when their length is known, and those it moved out of
        c10::Device device;
        at::Tensor col, val, earlier_col, earlier_val;
        std::exception_ptr failure;
    } taken{va.device};
    auto take = [](void *ctx, int64_t entries, int32_t **col, float **val) noexcept -> int {
        Taken &t = *static_cast<Taken *>(ctx);
        try {
            at::Tensor c = int_array(entries, t.device), v = float_array(entries, t.device);
            t.earlier_col = std::move(t.col), t.earlier_val = std::move(t.val);
            t.col = std::move(c), t.val = std::move(v);
            *col = ints(t.col), *val = floats(t.val);
            return NB200_OK;
        } catch (...) {
            t.failure = std::current_exception();
            return NB200_E_NOMEM;
        }
    };
    const int status = run({&va, &vb}, [&](void *stream) { return nb200_spgemm_f32_with(&a, &b, &c, take, &taken, stream); });
    if (status == NB200_E_NOMEM && taken.failure) std::rethrow_exception(taken.failure);
    check(status, where);
    at::Tensor &col = taken.col, &val = taken.val;
    if (!col.defined()) col = int_array(0, va.device), val = float_array(0, va.device);
    used(col, c.nnz);
    used(val, c.nnz);
    Result r(CSR);
    r.set(N_offsets, rp), r.set(N_indices, col), r.set(N_values, val);
    const int32_t d[2] = {c.rows, c.cols};
    r.dims<2>(d);
    return r.obj.release();
}

PyObject *coo_binary(coo2_fn fn, bool is_union, const char *where, PyObject *const *args) {
    for (int k = 0; k < 2; ++k) need_kind(args[k], COO, where, "COO_gpu");
    View va, vb;
    const nb200_coo a = view_coo(args[0], va), b = view_coo(args[1], vb);
    same_device(va, vb);
    const int64_t capacity = is_union ? (int64_t)a.nnz + b.nnz : std::min(a.nnz, b.nnz);
    at::Tensor i = int_array(capacity, va.device), j = int_array(capacity, va.device), val = float_array(capacity, va.device);
    nb200_coo z{a.rows, a.cols, 0, ints(i), ints(j), floats(val)};
    launch({&va, &vb}, where, [&](void *stream) { return fn(&a, &b, &z, capacity, stream); });
    used(i, z.nnz), used(j, z.nnz), used(val, z.nnz);
    Result r(COO);
    r.set(N_i, i), r.set(N_j, j), r.set(N_values, val);
    const int32_t d[2] = {z.rows, z.cols};
    r.dims<2>(d);
    return r.obj.release();
}

PyObject *coo_add(PyObject *const *args) { return coo_binary(nb200_coo_add_f32_into, true, "gpu_coo_add_f32", args); }
PyObject *coo_mul(PyObject *const *args) { return coo_binary(nb200_coo_mul_f32_into, false, "gpu_coo_mul_f32", args); }

PyObject *dcsr_binary(dcsr2_fn fn, bool is_union, const char *where, PyObject *const *args) {
    for (int k = 0; k < 2; ++k) need_kind(args[k], DCSR, where, "DCSR_gpu");
    View va, vb;
    const nb200_dcsr a = view_dcsr(args[0], va), b = view_dcsr(args[1], vb);
    same_device(va, vb);
    const int64_t cap_i = is_union ? std::min<int64_t>((int64_t)a.n_i + b.n_i, a.rows) : std::min(a.n_i, b.n_i);
    const int64_t capacity = is_union ? (int64_t)a.nnz + b.nnz : std::min(a.nnz, b.nnz);
    at::Tensor i = int_array(cap_i, va.device), jp = int_array(cap_i + 1, va.device), j = int_array(capacity, va.device), val = float_array(capacity, va.device);
    nb200_dcsr z{a.rows, a.cols, 0, 0, ints(i), ints(jp), ints(j), floats(val)};
    launch({&va, &vb}, where, [&](void *stream) { return fn(&a, &b, &z, cap_i, capacity, stream); });
    used(i, z.n_i), used(jp, (int64_t)z.n_i + 1), used(j, z.nnz), used(val, z.nnz);
    Result r(DCSR);
    r.set(N_i, i), r.set(N_jp, jp), r.set(N_j, j), r.set(N_values, val);
    const int32_t d[2] = {z.rows, z.cols};
    r.dims<2>(d);
    return r.obj.release();
}

PyObject *dcsr_add(PyObject *const *args) { return dcsr_binary(nb200_dcsr_add_f32_into, true, "gpu_dcsr_add_f32", args); }
PyObject *dcsr_mul(PyObject *const *args) { return dcsr_binary(nb200_dcsr_mul_f32_into, false, "gpu_dcsr_mul_f32", args); }

PyObject *coo3d_add(PyObject *const *args) {
    const char *where = "gpu_coo3d_add_f32";
    for (int k = 0; k < 2; ++k) need_kind(args[k], COO3, where, "COO3_gpu");
    View va, vb;
    const nb200_coo3 a = view_coo3(args[0], va), b = view_coo3(args[1], vb);
    same_device(va, vb);
    const int64_t capacity = (int64_t)a.nnz + b.nnz;
    at::Tensor i = int_array(capacity, va.device), j = int_array(capacity, va.device), k = int_array(capacity, va.device), val = float_array(capacity, va.device);
    nb200_coo3 z{};
    z.i = ints(i), z.j = ints(j), z.k = ints(k), z.val = floats(val);
    launch({&va, &vb}, where, [&](void *stream) { return nb200_coo3d_add_f32_into(&a, &b, &z, capacity, stream); });
    used(i, z.nnz), used(j, z.nnz), used(k, z.nnz), used(val, z.nnz);
    Result r(COO3);
    r.set(N_i, i), r.set(N_j, j), r.set(N_k, k), r.set(N_values, val);
    r.dims<3>(z.dims);
    return r.obj.release();
}

PyObject *csf_add(PyObject *const *args) {
    const char *where = "gpu_csf_add_f32";
    for (int k = 0; k < 2; ++k) need_kind(args[k], CSF3, where, "CSF3_gpu");
    View va, vb;
    const nb200_csf3 a = view_csf3(args[0], va), b = view_csf3(args[1], vb);
    same_device(va, vb);
    const int64_t cap_i = (int64_t)a.n_i + b.n_i, cap_j = (int64_t)a.n_j + b.n_j, cap_k = (int64_t)a.n_k + b.n_k;
    at::Tensor i = int_array(cap_i, va.device), jp = int_array(cap_i + 1, va.device), j = int_array(cap_j, va.device);
    at::Tensor kp = int_array(cap_j + 1, va.device), k = int_array(cap_k, va.device), val = float_array(cap_k, va.device);
    nb200_csf3 z{};
    z.i_idx = ints(i), z.j_ptr = ints(jp), z.j_idx = ints(j), z.k_ptr = ints(kp), z.k_idx = ints(k), z.val = floats(val);
    launch({&va, &vb}, where, [&](void *stream) { return nb200_csf_add_f32_into(&a, &b, &z, cap_i, cap_j, cap_k, stream); });
    used(i, z.n_i), used(jp, (int64_t)z.n_i + 1), used(j, z.n_j), used(kp, (int64_t)z.n_j + 1), used(k, z.n_k), used(val, z.n_k);
    Result r(CSF3);
    r.set(N_i, i), r.set(N_jp, jp), r.set(N_j, j), r.set(N_kp, kp), r.set(N_k, k), r.set(N_values, val);
    r.dims<3>(z.dims);
    return r.obj.release();
}

template <typename S, typename F>
PyObject *inner(Kind kind, const char *what, const char *where, PyObject *const *args, S (*view)(PyObject *, View &), F fn) {
    for (int k = 0; k < 2; ++k) need_kind(args[k], kind, where, what);
    View va, vb;
    const S a = view(args[0], va), b = view(args[1], vb);
    same_device(va, vb);
    at::Tensor z = float_array(1, va.device);
    launch({&va, &vb}, where, [&](void *stream) { return fn(&a, &b, floats(z), stream); });
    Result r(SCALAR);
    r.set(N_values, z);
    return r.obj.release();
}

PyObject *inner_prod(PyObject *const *args) { return inner(CSF3, "CSF3_gpu", "gpu_inner_prod_f32", args, view_csf3, nb200_inner_prod_f32); }
PyObject *inner_prod_coo(PyObject *const *args) { return inner(COO3, "COO3_gpu", "gpu_inner_prod_coo_f32", args, view_coo3, nb200_inner_prod_coo_f32); }

// ---- module --------------------------------------------------------------------------------

template <PyObject *(*OP)(PyObject *const *), int ARGS>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != ARGS) {
        PyErr_Format(PyExc_TypeError, "%d operands expected, %zd given", ARGS, n);
        return nullptr;
    }
    try {
        return OP(args);
    } catch (const PyFailure &) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// bind((CSR_gpu, COO_gpu, DCSR_gpu, COO3_gpu, CSF3_gpu, Scalar_gpu), check)
PyObject *bind(PyObject *, PyObject *args) {
    PyObject *classes, *check_fn;
    if (!PyArg_ParseTuple(args, "O!O", &PyTuple_Type, &classes, &check_fn)) return nullptr;
    if (PyTuple_GET_SIZE(classes) != KINDS) return PyErr_Format(PyExc_TypeError, "bind: %d classes expected", (int)KINDS);
    for (int k = 0; k < KINDS; ++k) {
        PyObject *c = PyTuple_GET_ITEM(classes, k);
        if (!PyType_Check(c)) return PyErr_Format(PyExc_TypeError, "bind: not a class");
        Py_INCREF(c);
        g_class[k] = reinterpret_cast<PyTypeObject *>(c);
    }
    Py_INCREF(check_fn);
    g_check = check_fn;
    Py_RETURN_NONE;
}

// turn_of(device, stream handle): identity of the lock by which calls there take turns (for tests)
PyObject *turn_of(PyObject *, PyObject *args) {
    int device;
    unsigned long long stream;
    if (!PyArg_ParseTuple(args, "iK", &device, &stream)) return nullptr;
    return PyLong_FromVoidPtr(&stream_lock(device, reinterpret_cast<void *>(stream)));
}

template <PyObject *(*OP)(PyObject *const *), int ARGS>
PyMethodDef op(const char *name) {
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<OP, ARGS>)), METH_FASTCALL, nullptr};
}

PyMethodDef g_methods[] = {
    {"bind", bind, METH_VARARGS, nullptr}, {"turn_of", turn_of, METH_VARARGS, nullptr},
    op<csr_add, 2>("csr_add"), op<csr_mul, 2>("csr_mul"), op<csr_add_3, 3>("csr_add_3"), op<spgemm, 2>("spgemm"),
    op<sssmm, 3>("sssmm"), op<coo3d_add, 2>("coo3d_add"), op<csf_add, 2>("csf_add"), op<coo_add, 2>("coo_add"),
    op<coo_mul, 2>("coo_mul"), op<coo_csr_add, 2>("coo_csr_add"), op<dcsr_add, 2>("dcsr_add"), op<dcsr_mul, 2>("dcsr_mul"),
    op<inner_prod, 2>("inner_prod"), op<inner_prod_coo, 2>("inner_prod_coo"),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    for (int k = 0; k < NAMES; ++k)
        if (!(g_name[k] = PyUnicode_InternFromString(NAME_TEXT[k]))) return nullptr;
    return PyModule_Create(&g_module);
}
