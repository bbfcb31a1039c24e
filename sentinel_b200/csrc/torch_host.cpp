// CPython module behind the Python entry points: checks the torch tensors, allocates the results, finds the scratch and
// calls the C ABI, all in native code.
//
// What it is for: on small problems the kernels of a call take 5-20 us and the host side sets the pace.  The same steps in
// Python (attribute lookups on every tensor, ctypes conversions, torch.empty through the dispatcher, current_stream) cost
// 20-25 us a call; here they cost about 3 us plus the launches.
//
// Every function takes exactly the positional arguments its Python caller has, and returns
//   a tuple of tensors   the call was made,
//   an int               the call was made and the library refused it (its status code), or
//   None                 something is not as the fast path wants it (a tensor that is not a contiguous CUDA tensor of the
//                        current device, shapes or types that do not match, an argument of another type): nothing has been
//                        done, and the Python code that follows names the error or makes the call itself.
//
// The library is the one ctypes has loaded: bind() receives the addresses of its entry points, so that another build of the
// same ABI can be put in its place.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "sntl_attn.h"

namespace {

decltype(&sntl_attn_fwd) p_fwd;
decltype(&sntl_attn_bwd) p_bwd;
decltype(&sntl_attn_cached_fwd) p_cached;
decltype(&sntl_attn_fwd_workspace_bytes) p_fwd_ws;
decltype(&sntl_attn_bwd_workspace_bytes) p_bwd_ws;
decltype(&sntl_attn_cached_fwd_workspace_bytes) p_cached_ws;
decltype(&sntl_attn_pack_heads) p_pack;
decltype(&sntl_attn_unpack_heads) p_unpack;

// Thrown away by guard(): the fast path does not apply.
struct Decline {};
struct PythonError {};   // a Python exception is set

// ---- arguments ----
int64_t as_int(PyObject* o)
{
    if (!PyLong_Check(o)) throw Decline{};   // (bool is an int)
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        throw Decline{};
    }
    return v;
}
int32_t as_i32(PyObject* o)
{
    const int64_t v = as_int(o);
    if (v < INT32_MIN || v > INT32_MAX) throw Decline{};
    return (int32_t)v;
}
float as_scale(PyObject* o, int64_t head_dim)
{
    if (o == Py_None) return head_dim > 0 ? (float)(1.0 / std::sqrt((double)head_dim)) : 0.0f;
    if (!PyFloat_Check(o)) throw Decline{};
    return (float)PyFloat_AS_DOUBLE(o);
}

// A contiguous CUDA tensor of the current device.
const at::Tensor& as_tensor(PyObject* o, c10::DeviceIndex device)
{
    if (!THPVariable_Check(o)) throw Decline{};
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || t.layout() != at::kStrided || !t.is_cuda() || t.device().index() != device || !t.is_contiguous() || t.is_neg() ||
        t.is_conj())
        throw Decline{};
    return t;
}
void want(bool ok)
{
    if (!ok) throw Decline{};
}

// A result: the caller's own tensor, which must be exactly what would have been allocated, or a new one.
at::Tensor result(PyObject* o, c10::IntArrayRef shape, at::ScalarType type, c10::DeviceIndex device)
{
    if (o == Py_None) return at::Tensor(at::detail::empty_cuda(shape, type, at::Device(at::kCUDA, device), std::nullopt));
    const at::Tensor& t = as_tensor(o, device);
    want(t.scalar_type() == type && t.sizes() == shape);
    return t;
}

template <typename... T>
PyObject* pack_tuple(const T&... t)
{
    PyObject* tuple = PyTuple_New(sizeof...(T));
    if (!tuple) throw PythonError{};
    Py_ssize_t i = 0;
    auto put = [&](const at::Tensor& x) { PyTuple_SET_ITEM(tuple, i++, THPVariable_Wrap(x)); };
    (put(t), ...);
    return tuple;
}

template <typename F>
PyObject* guard(F&& f)
{
    try {
        return f();
    } catch (const Decline&) {
        Py_RETURN_NONE;
    } catch (const PythonError&) {
        return nullptr;
    } catch (const c10::Error&) {
        Py_RETURN_NONE;   // no device, no memory: the Python code asks for the same things and raises torch's own exception
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// ---- scratch ----
// Grow-only, one buffer per (device, stream): calls on different streams may overlap on the GPU.  torch hands out streams
// from pools of 32 per device and priority, which bounds the number of entries.  The interpreter lock guards the map; it is given
// up during the launches, and the kernels of one call hand data to one another through the buffer, so calls of several threads on
// one stream are kept apart by the entry's own lock (taken without the interpreter lock: nothing waits for both).  A call keeps its
// own reference to the buffer while it launches; one that was replaced goes back to torch's allocator in stream order.
// A graph replays with the address it recorded.  A call that is being captured uses the buffer that is there (after a warm-up on
// this stream), which is then kept when a later call outgrows it; where there is none that is large enough it takes one of its
// own, which torch's allocator keeps for as long as the graph.
using WsKey = std::pair<int, void*>;
struct Scratch {
    at::Tensor buffer;
    std::mutex launching;
    bool recorded = false;            // a graph may hold the address of `buffer`
    std::vector<at::Tensor> kept;     // outgrown buffers of which that is true (one per growth at most)
};
Scratch& scratch(const WsKey& key)
{
    static auto* m = new std::map<WsKey, Scratch>;   // never destroyed: torch's allocator may be gone by then
    return (*m)[key];
}

struct Where {
    c10::DeviceIndex device = c10::cuda::current_device();
    void* stream = c10::cuda::getCurrentCUDAStream(device).stream();
};

// call(pointer to `bytes` of scratch, null for none), without the interpreter lock, as through ctypes
template <typename F>
int launch(const Where& at_, size_t bytes, F&& call)
{
    at::Tensor buffer;
    std::unique_lock<std::mutex> alone;
    auto allocate = [&] { return at::Tensor(at::detail::empty_cuda({(int64_t)bytes}, at::kByte, at::Device(at::kCUDA, at_.device), std::nullopt)); };
    if (bytes) {
        Scratch& s = scratch(WsKey(at_.device, at_.stream));
        const bool captured = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
        const bool fits = s.buffer.defined() && (size_t)s.buffer.numel() >= bytes;
        if (captured && !fits) {
            buffer = allocate();
        } else {
            if (!fits) {
                at::Tensor larger = allocate();
                if (s.recorded) s.kept.push_back(s.buffer);
                s.buffer = larger;
                s.recorded = false;
            }
            s.recorded = s.recorded || captured;
            buffer = s.buffer;
            alone = std::unique_lock<std::mutex>(s.launching, std::defer_lock);
        }
    }
    void* const p = bytes ? buffer.mutable_data_ptr() : nullptr;
    PyThreadState* state = PyEval_SaveThread();
    if (alone.mutex()) alone.lock();
    const int rc = call(p);
    if (alone.owns_lock()) alone.unlock();
    PyEval_RestoreThread(state);
    return rc;
}

int32_t dtype_code(const at::Tensor& t)
{
    if (t.scalar_type() == at::kBFloat16) return SNTL_DTYPE_BF16;
    want(t.scalar_type() == at::kFloat);
    return SNTL_DTYPE_F32;
}

sntl_attn_desc bhsd_desc(const at::Tensor& q, const at::Tensor& k, bool causal, float scale, int32_t flags, int32_t window, int32_t globals)
{
    want(q.dim() == 4 && k.dim() == 4 && k.size(0) == q.size(0) && k.size(3) == q.size(3));
    for (int i = 0; i < 4; ++i) want(q.size(i) <= INT32_MAX && k.size(i) <= INT32_MAX);
    sntl_attn_desc d{};
    d.dtype = dtype_code(q);
    d.layout = SNTL_LAYOUT_BHSD;
    d.batch = (int32_t)q.size(0);
    d.q_heads = (int32_t)q.size(1);
    d.kv_heads = (int32_t)k.size(1);
    d.seq_q = (int32_t)q.size(2);
    d.seq_kv = (int32_t)k.size(2);
    d.head_dim = (int32_t)q.size(3);
    d.scale = scale;
    d.causal = causal ? 1 : 0;
    d.flags = flags;
    d.window_size = window;
    d.global_tokens = globals;
    return d;
}
bool as_bool(PyObject* o)
{
    if (!PyBool_Check(o)) throw Decline{};
    return o == Py_True;
}

// ---- token-major calls ----
// (q, k, v, causal, scale, flags, out, lse, window, global_tokens)
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guard([&]() -> PyObject* {
        want(n == 10);
        const Where at_;
        const at::Tensor &q = as_tensor(a[0], at_.device), &k = as_tensor(a[1], at_.device), &v = as_tensor(a[2], at_.device);
        want(k.sizes() == v.sizes() && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type() && q.dim() == 4);
        const sntl_attn_desc d = bhsd_desc(q, k, as_bool(a[3]), as_scale(a[4], q.size(3)), as_i32(a[5]), as_i32(a[8]), as_i32(a[9]));
        const at::Tensor o = result(a[6], q.sizes(), q.scalar_type(), at_.device);
        const at::Tensor lse = result(a[7], q.sizes().slice(0, 3), at::kFloat, at_.device);
        const size_t bytes = p_fwd_ws(&d);
        const int rc = launch(at_, bytes, [&](void* ws) {
            return p_fwd(&d, q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), o.mutable_data_ptr(), (float*)lse.mutable_data_ptr(),
                         ws, bytes, at_.stream);
        });
        return rc == SNTL_OK ? pack_tuple(o, lse) : PyLong_FromLong(rc);
    });
}

// (q, k, v, o, lse, dout, causal, scale, flags, dq, dk, dv, window, global_tokens)
PyObject* backward(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guard([&]() -> PyObject* {
        want(n == 14);
        const Where at_;
        const at::Tensor &q = as_tensor(a[0], at_.device), &k = as_tensor(a[1], at_.device), &v = as_tensor(a[2], at_.device);
        const at::Tensor &o = as_tensor(a[3], at_.device), &lse = as_tensor(a[4], at_.device), &dout = as_tensor(a[5], at_.device);
        const auto type = q.scalar_type();
        want(q.dim() == 4 && o.sizes() == q.sizes() && dout.sizes() == q.sizes() && lse.sizes() == q.sizes().slice(0, 3));
        want(lse.scalar_type() == at::kFloat && k.sizes() == v.sizes());
        want(k.scalar_type() == type && v.scalar_type() == type && o.scalar_type() == type && dout.scalar_type() == type);
        const sntl_attn_desc d = bhsd_desc(q, k, as_bool(a[6]), as_scale(a[7], q.size(3)), as_i32(a[8]), as_i32(a[12]), as_i32(a[13]));
        const at::Tensor dq = result(a[9], q.sizes(), type, at_.device), dk = result(a[10], k.sizes(), type, at_.device);
        const at::Tensor dv = result(a[11], v.sizes(), type, at_.device);
        const size_t bytes = p_bwd_ws(&d);
        const int rc = launch(at_, bytes, [&](void* ws) {
            return p_bwd(&d, q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), o.const_data_ptr(), (const float*)lse.const_data_ptr(),
                         dout.const_data_ptr(), dq.mutable_data_ptr(), dk.mutable_data_ptr(), dv.mutable_data_ptr(),
                         ws, bytes, at_.stream);
        });
        return rc == SNTL_OK ? pack_tuple(dq, dk, dv) : PyLong_FromLong(rc);
    });
}

// (q, k_cache, v_cache, cache_length, scale, flags, out, lse, window, global_tokens)
PyObject* cached_forward(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guard([&]() -> PyObject* {
        want(n == 10);
        const Where at_;
        const at::Tensor &q = as_tensor(a[0], at_.device), &k = as_tensor(a[1], at_.device), &v = as_tensor(a[2], at_.device);
        want(k.sizes() == v.sizes() && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type() && q.dim() == 4);
        sntl_attn_desc d = bhsd_desc(q, k, true, as_scale(a[4], q.size(3)), as_i32(a[5]), as_i32(a[8]), as_i32(a[9]));
        const int32_t capacity = d.seq_kv;
        d.seq_kv = as_i32(a[3]);
        const at::Tensor o = result(a[6], q.sizes(), q.scalar_type(), at_.device);
        const at::Tensor lse = result(a[7], q.sizes().slice(0, 3), at::kFloat, at_.device);
        const size_t bytes = p_cached_ws(&d, capacity);
        const int rc = launch(at_, bytes, [&](void* ws) {
            return p_cached(&d, q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), capacity, o.mutable_data_ptr(),
                            (float*)lse.mutable_data_ptr(), ws, bytes, at_.stream);
        });
        return rc == SNTL_OK ? pack_tuple(o, lse) : PyLong_FromLong(rc);
    });
}

// ---- feature-major calls ----
// a matrix argument: fp32, two-dimensional
const at::Tensor& as_matrix(PyObject* o, c10::DeviceIndex device)
{
    const at::Tensor& t = as_tensor(o, device);
    want(t.dim() == 2 && t.scalar_type() == at::kFloat && t.size(0) <= INT32_MAX && t.size(1) <= INT32_MAX);
    return t;
}
// the tail both calls share: headCount, headDimension, scale, causal, columnStart, columnCount, packCount, windowSize,
// globalTokenCount, flags
constexpr int kMatrixTail = 10;
sntl_attn_desc matrix_desc(const at::Tensor& q, const at::Tensor& k, PyObject* const* a)
{
    const int32_t heads = as_i32(a[0]), dim = as_i32(a[1]), start = as_i32(a[4]);
    int32_t count = as_i32(a[5]), packs = as_i32(a[6]);
    want(q.numel() > 0 && k.numel() > 0 && heads > 0 && dim > 0 && q.size(0) == (int64_t)heads * dim && k.size(0) % dim == 0);
    const int32_t kv = (int32_t)(k.size(0) / dim), stride = (int32_t)q.size(1);
    want(kv > 0 && heads % kv == 0 && k.size(1) == stride && PyFloat_Check(a[2]));
    if (packs <= 0) packs = 1;
    if (count <= 0) count = stride - start;
    want(start >= 0 && count > 0 && (int64_t)start + (int64_t)packs * count <= stride);
    sntl_attn_desc d{};
    d.dtype = SNTL_DTYPE_F32;
    d.layout = SNTL_LAYOUT_SENTINEL;
    d.batch = packs;
    d.q_heads = heads;
    d.kv_heads = kv;
    d.seq_q = d.seq_kv = count;
    d.head_dim = dim;
    d.scale = (float)PyFloat_AS_DOUBLE(a[2]);
    d.causal = as_bool(a[3]) ? 1 : 0;
    d.stride_columns = stride;
    d.column_start = start;
    d.window_size = as_i32(a[7]);
    d.global_tokens = as_i32(a[8]);
    d.flags = as_i32(a[9]);
    return d;
}

// (query, key, value, out, logSumExp) + tail; the results are the caller's
PyObject* matrix_forward(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guard([&]() -> PyObject* {
        want(n == 5 + kMatrixTail);
        const Where at_;
        const at::Tensor &q = as_matrix(a[0], at_.device), &k = as_matrix(a[1], at_.device), &v = as_matrix(a[2], at_.device);
        const at::Tensor &o = as_matrix(a[3], at_.device), &lse = as_matrix(a[4], at_.device);
        const sntl_attn_desc d = matrix_desc(q, k, a + 5);
        want(k.sizes() == v.sizes() && o.sizes() == q.sizes() && lse.size(0) == d.q_heads && lse.size(1) == d.stride_columns);
        const size_t bytes = p_fwd_ws(&d);
        const int rc = launch(at_, bytes, [&](void* ws) {
            return p_fwd(&d, q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), o.mutable_data_ptr(), (float*)lse.mutable_data_ptr(),
                         ws, bytes, at_.stream);
        });
        return rc == SNTL_OK ? pack_tuple(o, lse) : PyLong_FromLong(rc);
    });
}

// (query, key, value, out, logSumExp, outGradient, queryGradient, keyGradient, valueGradient) + tail
PyObject* matrix_backward(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guard([&]() -> PyObject* {
        want(n == 9 + kMatrixTail);
        const Where at_;
        const at::Tensor &q = as_matrix(a[0], at_.device), &k = as_matrix(a[1], at_.device), &v = as_matrix(a[2], at_.device);
        const at::Tensor &o = as_matrix(a[3], at_.device), &lse = as_matrix(a[4], at_.device), &g = as_matrix(a[5], at_.device);
        const at::Tensor &dq = as_matrix(a[6], at_.device), &dk = as_matrix(a[7], at_.device), &dv = as_matrix(a[8], at_.device);
        const sntl_attn_desc d = matrix_desc(q, k, a + 9);
        want(k.sizes() == v.sizes() && o.sizes() == q.sizes() && g.sizes() == q.sizes() && dq.sizes() == q.sizes());
        want(dk.sizes() == k.sizes() && dv.sizes() == k.sizes() && lse.size(0) == d.q_heads && lse.size(1) == d.stride_columns);
        const size_t bytes = p_bwd_ws(&d);
        const int rc = launch(at_, bytes, [&](void* ws) {
            return p_bwd(&d, q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), o.const_data_ptr(), (const float*)lse.const_data_ptr(),
                         g.const_data_ptr(), dq.mutable_data_ptr(), dk.mutable_data_ptr(), dv.mutable_data_ptr(),
                         ws, bytes, at_.stream);
        });
        return rc == SNTL_OK ? pack_tuple(dq, dk, dv) : PyLong_FromLong(rc);
    });
}

// ---- boundary conversions ----
struct Tables {
    const float *cos = nullptr, *sin = nullptr;
    int32_t positions = 0;
};
Tables as_tables(PyObject* c, PyObject* s, int64_t head_dim, c10::DeviceIndex device)
{
    Tables t;
    if (c == Py_None && s == Py_None) return t;
    const at::Tensor &tc = as_matrix(c, device), &ts = as_matrix(s, device);
    want(tc.sizes() == ts.sizes() && tc.size(1) == head_dim / 2);
    t.cos = (const float*)tc.const_data_ptr();
    t.sin = (const float*)ts.const_data_ptr();
    t.positions = (int32_t)tc.size(0);
    return t;
}

// (matrix, batch, heads, seq, head_dim, column_start, cos_table, sin_table, position_offset, out)
PyObject* pack_heads(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guard([&]() -> PyObject* {
        want(n == 10);
        const Where at_;
        const at::Tensor& m = as_matrix(a[0], at_.device);
        const int32_t batch = as_i32(a[1]), heads = as_i32(a[2]), seq = as_i32(a[3]), dim = as_i32(a[4]);
        want(batch > 0 && heads > 0 && seq > 0 && dim > 0 && m.size(0) == (int64_t)heads * dim);
        const Tables t = as_tables(a[6], a[7], dim, at_.device);
        const int32_t start = as_i32(a[5]), offset = as_i32(a[8]);
        const int64_t shape[4] = {batch, heads, seq, dim};
        const at::Tensor out = result(a[9], shape, at::kBFloat16, at_.device);
        const int rc = launch(at_, 0, [&](void*) {
            return p_pack((const float*)m.const_data_ptr(), out.mutable_data_ptr(), batch, heads, seq, dim, (int32_t)m.size(1), start, t.cos,
                          t.sin, offset, t.positions, at_.stream);
        });
        return rc == SNTL_OK ? THPVariable_Wrap(out) : PyLong_FromLong(rc);
    });
}

// (tensor, matrix, column_start, cos_table, sin_table, position_offset, inverse)
PyObject* unpack_heads(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    return guard([&]() -> PyObject* {
        want(n == 7);
        const Where at_;
        const at::Tensor &x = as_tensor(a[0], at_.device), &m = as_matrix(a[1], at_.device);
        want(x.scalar_type() == at::kBFloat16 && x.dim() == 4 && m.size(0) == x.size(1) * x.size(3));
        for (int i = 0; i < 4; ++i) want(x.size(i) <= INT32_MAX);
        const Tables t = as_tables(a[3], a[4], x.size(3), at_.device);
        const int32_t start = as_i32(a[2]), offset = as_i32(a[5]), inverse = as_bool(a[6]) ? 1 : 0;
        const int rc = launch(at_, 0, [&](void*) {
            return p_unpack(x.const_data_ptr(), (float*)m.mutable_data_ptr(), (int32_t)x.size(0), (int32_t)x.size(1), (int32_t)x.size(2),
                            (int32_t)x.size(3), (int32_t)m.size(1), start, t.cos, t.sin, offset, t.positions, inverse, at_.stream);
        });
        if (rc != SNTL_OK) return PyLong_FromLong(rc);
        Py_INCREF(a[1]);
        return a[1];
    });
}

// bind(addresses): in the order of the pointers below
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n)
{
    if (n != 8) {
        PyErr_SetString(PyExc_TypeError, "bind() takes the addresses of 8 entry points");
        return nullptr;
    }
    void* p[8];
    for (int i = 0; i < 8; ++i)
        if (!(p[i] = PyLong_AsVoidPtr(a[i]))) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry point");
            return nullptr;
        }
    p_fwd = (decltype(p_fwd))p[0];
    p_bwd = (decltype(p_bwd))p[1];
    p_cached = (decltype(p_cached))p[2];
    p_fwd_ws = (decltype(p_fwd_ws))p[3];
    p_bwd_ws = (decltype(p_bwd_ws))p[4];
    p_cached_ws = (decltype(p_cached_ws))p[5];
    p_pack = (decltype(p_pack))p[6];
    p_unpack = (decltype(p_unpack))p[7];
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)())bind, METH_FASTCALL, nullptr},
    {"forward", (PyCFunction)(void (*)())forward, METH_FASTCALL, nullptr},
    {"backward", (PyCFunction)(void (*)())backward, METH_FASTCALL, nullptr},
    {"cached_forward", (PyCFunction)(void (*)())cached_forward, METH_FASTCALL, nullptr},
    {"matrix_forward", (PyCFunction)(void (*)())matrix_forward, METH_FASTCALL, nullptr},
    {"matrix_backward", (PyCFunction)(void (*)())matrix_backward, METH_FASTCALL, nullptr},
    {"pack_heads", (PyCFunction)(void (*)())pack_heads, METH_FASTCALL, nullptr},
    {"unpack_heads", (PyCFunction)(void (*)())unpack_heads, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_sntl_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// Nothing else notices when torch has been exchanged since the build: its C++ interface is not stable from version to version.
bool torch_is_the_one_built_for()
{
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* version = torch ? PyObject_GetAttrString(torch, "__version__") : nullptr;
    PyObject* text = version ? PyObject_Str(version) : nullptr;
    const char* running = text ? PyUnicode_AsUTF8(text) : nullptr;
    const bool same = running && std::strcmp(running, SNTL_TORCH_VERSION) == 0;
    if (running && !same) PyErr_Format(PyExc_ImportError, "built for torch %s, running with %s", SNTL_TORCH_VERSION, running);
    Py_XDECREF(text);
    Py_XDECREF(version);
    Py_XDECREF(torch);
    return same;
}

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__sntl_host()
{
    return torch_is_the_one_built_for() ? PyModule_Create(&module) : nullptr;
}
