// binding.cpp -- the per-call half of the Python package as a CPython extension (module `_binding`): tensor checks, result
// allocation, stream lookup and the call into libtllm.so (include/tllm.h), without a Python-level attribute walk or a
// ctypes argument conversion per call.
//
// A decode product runs 3 to 10 us on the GPU; the same call through ctypes took 16 us of host time (info struct to dict,
// device context manager, stream object, torch.empty, nine converted arguments), so a decode loop that is not captured in
// a graph was bound by the host.  Here a call costs the checks (tens of ns), one allocation from torch's caching
// allocator and the launch.  Only host plumbing lives here; kernels, dispatch and handles are libtllm's.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/Parallel.h>
#include <ATen/RedispatchFunctions.h>
#include <ATen/core/CachingHostAllocator.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cuda_runtime.h>

#include <algorithm>
#include <exception>
#include <string>

#include "../../include/tllm.h"

namespace {

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return TLLM_F32;
        case at::kHalf: return TLLM_F16;
        case at::kBFloat16: return TLLM_BF16;
        case at::kChar: return TLLM_I8;
        case at::kInt: return TLLM_I32;
        default: return -1;
    }
}

PyObject* raise(const std::string& msg) {
    PyErr_SetString(PyExc_RuntimeError, msg.c_str());
    return nullptr;
}

PyObject* raise_rc(const char* what, int rc) {
    const char* m = tllm_last_error();
    return raise(std::string(what) + ": " + (m && *m ? m : "error") + " (code " + std::to_string(rc) + ")");
}

const at::Tensor* tensor_of(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

bool int_of(PyObject* o, long long* v) {
    *v = PyLong_AsLongLong(o);
    return !(*v == -1 && PyErr_Occurred());
}

// makes `device` current for the scope of a call; nothing when it already is
struct DeviceScope {
    c10::cuda::OptionalCUDAGuard g;
    explicit DeviceScope(c10::DeviceIndex device) {
        if (c10::cuda::current_device() != device) g.set_index(device);
    }
};

// the interpreter is free for other threads until the end of the scope, exceptions included
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

std::string shape_text(const at::Tensor& t) {
    std::string s = "torch.Size([";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + "])";
}

#define NEED_ARGS(n, who)                                                        \
    if (nargs != (n)) {                                                           \
        PyErr_SetString(PyExc_TypeError, who ": wrong number of arguments");      \
        return nullptr;                                                           \
    }
// C++ exceptions (allocation failure, bad stream) become Python errors
#define BINDING_TRY try {
#define BINDING_CATCH                  \
    }                                  \
    catch (const std::exception& e) {  \
        return raise(e.what());        \
    }

// matmul(handle, x, out | None, col_major, device, inners, columns) -> tensor
PyObject* matmul(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    NEED_ARGS(7, "matmul")
    BINDING_TRY
    long long handle, device, inners, columns;
    if (!int_of(a[0], &handle) || !int_of(a[4], &device) || !int_of(a[5], &inners) || !int_of(a[6], &columns)) return nullptr;
    const at::Tensor* xp = tensor_of(a[1]);
    if (!xp) return raise("matmul expects a tensor");
    const int col_major = PyObject_IsTrue(a[3]);
    if (col_major < 0) return nullptr;
    if (!xp->is_cuda() || xp->get_device() != device) return raise("activation must be on the CUDA device that holds the packed weight");
    if (xp->dim() != 2) return raise("matmul expects a 2-D activation");
    at::Tensor xc;
    if (!xp->is_contiguous()) xc = xp->contiguous(), xp = &xc;
    const int64_t rows = xp->size(col_major ? 1 : 0);
    if (xp->size(col_major ? 0 : 1) != inners) return raise("activation has " + shape_text(*xp) + " but the weight has " + std::to_string(inners) + " inners");
    if (rows > INT32_MAX) return raise("matmul: too many rows");
    const at::ScalarType xt = xp->scalar_type(), yt = xt == at::kChar ? at::kInt : xt;
    const int xcode = dtype_code(xt);
    if (xcode < 0) {
        PyErr_SetString(PyExc_KeyError, c10::toString(xt));
        return nullptr;
    }
    DeviceScope scope((c10::DeviceIndex)device);
    at::Tensor y;
    if (a[2] == Py_None) {
        y = at::empty({rows, columns}, xp->options().dtype(yt));
    } else {
        const at::Tensor* op = tensor_of(a[2]);
        if (!op) return raise("out must be a tensor");
        const at::ScalarType ot = op->scalar_type();
        if ((ot != yt && !(ot == at::kFloat && yt != at::kInt)) || op->dim() != 2 || op->size(0) != rows || op->size(1) != columns || !op->is_contiguous())
            return raise("out has the wrong dtype, shape or strides");
        y = *op;
    }
    void* st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    const void* X = xp->const_data_ptr();
    void* Y = y.data_ptr();
    const int ycode = dtype_code(y.scalar_type());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = tllm_spmm((tllm_weight*)handle, X, xcode, col_major ? TLLM_COL_MAJOR : TLLM_ROW_MAJOR, (int)rows, Y, ycode, st);
    Py_END_ALLOW_THREADS
    if (rc) return raise_rc("tllm_spmm", rc);
    if (a[2] != Py_None) {
        Py_INCREF(a[2]);
        return a[2];
    }
    return THPVariable_Wrap(std::move(y));
    BINDING_CATCH
}

// matmul_host(handle, x, x_code, x_col_major, rows, y, y_code, y_col_major, device): x and y are C-contiguous buffers, y writable
// and of rows * columns elements.  Copies in, runs, copies out, synchronises.
//
// The bus moves page-locked memory at 50 GB/s; what is pageable goes through the one thread that the driver copies it with (1 MB in 82 us instead of 20,
// a result of 4 MB in 257 instead of 86).  Buffers of some size therefore go through blocks of torch's page-locked cache, which torch's threads
// fill and empty, a result piece by piece while the next one is on the bus; the blocks are back in the cache when the call returns, and only
// calls that run at the same time need more than two.  (256 columns of fp32, 1024 x 4096, sixteen threads: 214 us, 288 with only the result staged, and
// in one piece; 2048 x 8192 377 and 504.  Pieces of 1 MB 217 and 383, of 2 MB 236 and 417.)
constexpr int64_t STAGE_X_FROM = 128 << 10, STAGE_FROM = 256 << 10, STAGE_TO = 16 << 20, STAGE_PART = 512 << 10;
// Straight to the CPU's copy: a dispatch mode of the caller's has no part in it.  torch deals out equal numbers of elements, 32768 or more to a thread, so that bytes
// would start anywhere for five to seven threads: these get elements as wide as leave work for four of them.  (64 rows of fp32, 4096 x 512: 97 us, 119 to 132 in bytes, 128
// unstaged; 64 on 2048 x 2048 89, 95 to 105, 107.  Twelve threads are better off with bytes.)
void copy_bytes(char* to, const char* from, int64_t n) {
    const int threads = at::get_num_threads();
    int64_t e = threads > 4 && threads < 8 ? 8 : 1;
    while (e > 1 && (n / e < 4 * 32768 || ((uintptr_t)to | (uintptr_t)from | (uintptr_t)n) % e != 0)) e /= 2;
    const at::ScalarType type = e == 8 ? at::kLong : e == 4 ? at::kInt : e == 2 ? at::kShort : at::kByte;
    at::Tensor t = at::from_blob(to, {n / e}, type);
    at::redispatch::copy_(c10::DispatchKeySet(c10::DispatchKey::CPU), t, at::from_blob(const_cast<char*>(from), {n / e}, type));
}
PyObject* matmul_host(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    NEED_ARGS(9, "matmul_host")
    BINDING_TRY
    long long v[9];
    for (int i = 0; i < 9; ++i)
        if (i != 1 && i != 5 && !int_of(a[i], &v[i])) return nullptr;
    struct Buffer {
        Py_buffer b{};
        bool held = false;
        bool get(PyObject* o, int flags) { return held = PyObject_GetBuffer(o, &b, flags) == 0; }
        ~Buffer() {
            if (held) PyBuffer_Release(&b);
        }
    } x, y;
    if (!x.get(a[1], PyBUF_C_CONTIGUOUS) || !y.get(a[5], PyBUF_C_CONTIGUOUS | PyBUF_WRITABLE)) return nullptr;
    DeviceScope scope((c10::DeviceIndex)v[8]);
    const int64_t bytes = y.b.len, x_bytes = x.b.len;
    const bool threads = at::get_num_threads() >= 4;
    c10::DataPtr x_stage, y_stage;
    if (threads && x_bytes >= STAGE_X_FROM && x_bytes <= STAGE_TO) x_stage = at::getHostAllocator(at::kCUDA)->allocate((size_t)x_bytes);
    if (threads && bytes >= STAGE_FROM && bytes <= STAGE_TO) y_stage = at::getHostAllocator(at::kCUDA)->allocate((size_t)bytes);
    struct Result {
        char *to, *from;
        std::exception_ptr failed;
    } out{(char*)y.b.buf, (char*)y_stage.get(), nullptr};
    const auto ready = [](void* a, size_t b, size_t e) {
        Result* r = (Result*)a;
        try {
            copy_bytes(r->to + b, r->from + b, (int64_t)(e - b));
        } catch (...) {
            r->failed = std::current_exception();
        }
    };
    int rc = 0;
    {
        NoGil no_gil;
        const void* X = x.b.buf;
        if (x_stage.get()) {
            copy_bytes((char*)x_stage.get(), (const char*)X, x_bytes);
            X = x_stage.get();
        }
        const int xl = v[3] ? TLLM_COL_MAJOR : TLLM_ROW_MAJOR, yl = v[7] ? TLLM_COL_MAJOR : TLLM_ROW_MAJOR;
        if (out.from) {
            const int parts = (int)std::min<int64_t>(TLLM_HOST_PARTS, (bytes + STAGE_PART - 1) / STAGE_PART);
            rc = tllm_spmm_host_parts((tllm_weight*)v[0], X, (int)v[2], xl, (int)v[4], out.from, (int)v[6], yl, parts, ready, &out);
        } else rc = tllm_spmm_host((tllm_weight*)v[0], X, (int)v[2], xl, (int)v[4], out.to, (int)v[6], yl);
    }
    if (rc) return raise_rc("tllm_spmm_host", rc);
    if (out.failed) std::rethrow_exception(out.failed);
    Py_RETURN_NONE;
    BINDING_CATCH
}

// mlp_forward(handle, x, out | None, h | None, hidden) -> tensor
PyObject* mlp_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    NEED_ARGS(5, "mlp_forward")
    BINDING_TRY
    long long handle, hidden;
    if (!int_of(a[0], &handle) || !int_of(a[4], &hidden)) return nullptr;
    const at::Tensor* xp = tensor_of(a[1]);
    if (!xp || !xp->is_cuda() || xp->dim() != 2 || xp->size(1) != hidden) return raise("PackedMLP.forward expects a 2-D CUDA activation [rows, hidden]");
    at::Tensor xc;
    if (!xp->is_contiguous()) xc = xp->contiguous(), xp = &xc;
    const int64_t rows = xp->size(0);
    if (rows > INT32_MAX) return raise("PackedMLP.forward: too many rows");
    const at::ScalarType xt = xp->scalar_type();
    const int xcode = dtype_code(xt);
    if (xcode < 0) {
        PyErr_SetString(PyExc_KeyError, c10::toString(xt));
        return nullptr;
    }
    DeviceScope scope(xp->get_device());
    at::Tensor y, h;
    if (a[2] == Py_None) {
        y = at::empty({rows, hidden}, xp->options());
    } else {
        const at::Tensor* op = tensor_of(a[2]);
        if (!op) return raise("out must be a tensor");
        if ((op->scalar_type() != xt && op->scalar_type() != at::kFloat) || op->dim() != 2 || op->size(0) != rows || op->size(1) != hidden || !op->is_contiguous())
            return raise("out has the wrong dtype, shape or strides");
        y = *op;
    }
    if (a[3] != Py_None) {
        const at::Tensor* hp = tensor_of(a[3]);
        if (!hp) return raise("h must be a tensor");
        h = *hp;
    }
    void* st = c10::cuda::getCurrentCUDAStream(xp->get_device()).stream();
    const void* X = xp->const_data_ptr();
    void *Y = y.data_ptr(), *H = h.defined() ? h.data_ptr() : nullptr;
    const int ycode = dtype_code(y.scalar_type());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = tllm_mlp_forward_ex((tllm_mlp*)handle, X, xcode, (int)rows, Y, ycode, H, st);
    Py_END_ALLOW_THREADS
    if (rc) return raise_rc("tllm_mlp_forward", rc);
    if (a[2] != Py_None) {
        Py_INCREF(a[2]);
        return a[2];
    }
    return THPVariable_Wrap(std::move(y));
    BINDING_CATCH
}

// causal_attention(qkv [batch * rows, (heads + 2 * kv_heads) * head_dim], batch, rows, heads, kv_heads, head_dim) -> [batch * rows, heads * head_dim]
PyObject* causal_attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    NEED_ARGS(6, "causal_attention")
    BINDING_TRY
    long long v[6];
    for (int i = 1; i < 6; ++i)
        if (!int_of(a[i], &v[i])) return nullptr;
    const at::Tensor* x = tensor_of(a[0]);
    if (!x || !x->is_cuda() || x->dim() != 2 || !x->is_contiguous() || x->size(0) != v[1] * v[2] || x->size(1) != (v[3] + 2 * v[4]) * v[5])
        return raise("causal_attention expects a contiguous CUDA tensor [batch * rows, (heads + 2 * kv_heads) * head_dim]");
    DeviceScope scope(x->get_device());
    at::Tensor y = at::empty({x->size(0), v[3] * v[5]}, x->options());
    void* st = c10::cuda::getCurrentCUDAStream(x->get_device()).stream();
    const int rc = tllm_causal_attention(x->const_data_ptr(), y.data_ptr(), dtype_code(x->scalar_type()), (int)v[1], (int)v[2], (int)v[3], (int)v[4], (int)v[5], st);
    if (rc) return raise_rc("tllm_causal_attention", rc);
    return THPVariable_Wrap(std::move(y));
    BINDING_CATCH
}

// decode_attention(qkv [rows, (heads + 2 * kv_heads) * head_dim], k_cache, v_cache [>= rows, kv_heads, positions, head_dim], heads, len) -> [rows, heads * head_dim];
// the caches' position len is written
PyObject* decode_attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    NEED_ARGS(5, "decode_attention")
    BINDING_TRY
    long long heads, len;
    if (!int_of(a[3], &heads) || !int_of(a[4], &len)) return nullptr;
    const at::Tensor *x = tensor_of(a[0]), *k = tensor_of(a[1]), *v = tensor_of(a[2]);
    if (!x || !k || !v || !x->is_cuda() || x->dim() != 2 || !x->is_contiguous() || k->dim() != 4 || !k->is_contiguous() || !v->is_contiguous() || k->sizes() != v->sizes() ||
        k->device() != x->device() || v->device() != x->device() || k->scalar_type() != x->scalar_type() || v->scalar_type() != x->scalar_type() || k->size(0) < x->size(0) ||
        len < 0 || len >= k->size(2) || x->size(1) != (heads + 2 * k->size(1)) * k->size(3))
        return raise("decode_attention expects contiguous CUDA tensors qkv [rows, (heads + 2 * kv_heads) * head_dim] and caches [>= rows, kv_heads, > len, head_dim] of one type");
    DeviceScope scope(x->get_device());
    at::Tensor y = at::empty({x->size(0), heads * k->size(3)}, x->options());
    void* st = c10::cuda::getCurrentCUDAStream(x->get_device()).stream();
    const int rc = tllm_decode_attention(x->const_data_ptr(), k->data_ptr(), v->data_ptr(), y.data_ptr(), dtype_code(x->scalar_type()), (int)x->size(0), (int)heads, (int)k->size(1),
                                         (int)k->size(3), (int)len, k->stride(0), k->stride(1), st);
    if (rc) return raise_rc("tllm_decode_attention", rc);
    return THPVariable_Wrap(std::move(y));
    BINDING_CATCH
}

// ter_spmm(X, row_idx, col_off, tile_idx | None, batch, rows, columns, inners, uniformed, padded, scale, out | None, tile_k, prepare) -> tensor
// prepare: outside a stream capture the arrays are repacked first (tllm_ter_spmm_prepare), once every check has passed
PyObject* ter_spmm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    NEED_ARGS(14, "ter_spmm")
    BINDING_TRY
    const at::Tensor *xp = tensor_of(a[0]), *ip = tensor_of(a[1]), *op = tensor_of(a[2]);
    long long batch, rows, columns, inners, tile_k;
    if (!int_of(a[4], &batch) || !int_of(a[5], &rows) || !int_of(a[6], &columns) || !int_of(a[7], &inners) || !int_of(a[12], &tile_k)) return nullptr;
    const int uniformed = PyObject_IsTrue(a[8]), padded = PyObject_IsTrue(a[9]), prepare = PyObject_IsTrue(a[13]);
    const double scale = PyFloat_AsDouble(a[10]);
    if (uniformed < 0 || padded < 0 || prepare < 0 || (scale == -1.0 && PyErr_Occurred())) return nullptr;
    const at::Tensor* three[3] = {xp, ip, op};
    const char* names[3] = {"X", "row indices", "col offsets"};
    for (int i = 0; i < 3; ++i)
        if (!three[i] || !three[i]->is_cuda()) return raise(std::string("ter_spmm: ") + names[i] + " must be a CUDA tensor");
    if (ip->scalar_type() != at::kShort) return raise("ter_spmm: row indices must be int16");
    if (op->scalar_type() != at::kInt) return raise("ter_spmm: col offsets must be int32");
    const at::ScalarType xt = xp->scalar_type(), yt = xt == at::kChar ? at::kInt : xt;
    if (xt != at::kFloat && xt != at::kHalf && xt != at::kBFloat16 && xt != at::kChar)
        return raise(std::string("ter_spmm: unsupported activation dtype torch.") + c10::toString(xt));
    at::Tensor xc;
    if (!xp->is_contiguous()) xc = xp->contiguous(), xp = &xc;
    const int64_t d = xp->dim();
    const int layout = d >= 1 && xp->size(d - 1) == inners ? TLLM_ROW_MAJOR : TLLM_COL_MAJOR;
    if (layout == TLLM_COL_MAJOR && !(d >= 2 && xp->size(d - 2) == inners))
        return raise("ter_spmm: activation of shape " + shape_text(*xp) + " has no dimension of " + std::to_string(inners) + " inners");
    if (batch > 0 && xp->numel() != batch * rows * inners) return raise("ter_spmm: activation size does not match batch_size*rows*inners");
    if (tile_k <= 0) return raise("ter_spmm: TILE_K must be positive");
    const int64_t tiles = (inners + tile_k - 1) / tile_k;
    if (op->numel() != columns * tiles * 4) return raise("ter_spmm: col offsets do not have columns*ceil(inners/TILE_K)*4 entries");
    DeviceScope scope(xp->get_device());
    at::Tensor y;
    if (a[11] == Py_None) {
        y = at::empty({batch, rows, columns}, xp->options().dtype(yt));
    } else {
        const at::Tensor* o = tensor_of(a[11]);
        if (!o || o->scalar_type() != yt || o->numel() != batch * rows * columns || !o->is_contiguous())
            return raise("ter_spmm: out has the wrong dtype, size or strides");
        y = *o;
    }
    if (batch != 0) {   // the reference launches nothing for an empty batch (TernaryLinear.py:168)
        const at::Tensor* tp = tensor_of(a[3]);
        const int16_t* tile_ptr = tp && tp->numel() ? (const int16_t*)tp->const_data_ptr() : nullptr;
        void* st = c10::cuda::getCurrentCUDAStream(xp->get_device()).stream();
        const void* X = xp->const_data_ptr();
        void* Y = y.data_ptr();
        const int xcode = dtype_code(xt), ycode = dtype_code(yt);
        const int16_t* idx = (const int16_t*)ip->const_data_ptr();
        const int32_t* off = (const int32_t*)op->const_data_ptr();
        int rc;
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (prepare) C10_CUDA_CHECK(cudaStreamIsCapturing((cudaStream_t)st, &capture));
        if (prepare && capture == cudaStreamCaptureStatusNone) {
            DeviceScope there(ip->get_device());
            Py_BEGIN_ALLOW_THREADS
            rc = tllm_ter_spmm_prepare(idx, off, (int)columns, (int)inners, (int)tile_k);
            Py_END_ALLOW_THREADS
            if (rc) return raise_rc("ter_spmm.prepare", rc);
        }
        Py_BEGIN_ALLOW_THREADS
        rc = tllm_ter_spmm(X, xcode, layout, idx, off, tile_ptr, Y, ycode, (int)batch, (int)rows, (int)columns, (int)inners, (int)tile_k, (float)scale,
                           uniformed, padded, st);
        Py_END_ALLOW_THREADS
        if (rc) return raise_rc("ter_spmm", rc);
    }
    if (a[11] != Py_None) {
        Py_INCREF(a[11]);
        return a[11];
    }
    return THPVariable_Wrap(std::move(y));
    BINDING_CATCH
}

PyMethodDef methods[] = {
    {"matmul", (PyCFunction)(void (*)(void))matmul, METH_FASTCALL, "matmul(handle, x, out, col_major, device, inners, columns)"},
    {"matmul_host", (PyCFunction)(void (*)(void))matmul_host, METH_FASTCALL,
     "matmul_host(handle, x, x_code, x_col_major, rows, y, y_code, y_col_major, device)"},
    {"mlp_forward", (PyCFunction)(void (*)(void))mlp_forward, METH_FASTCALL, "mlp_forward(handle, x, out, h, hidden)"},
    {"decode_attention", (PyCFunction)(void (*)(void))decode_attention, METH_FASTCALL, "decode_attention(qkv, k_cache, v_cache, heads, len)"},
    {"causal_attention", (PyCFunction)(void (*)(void))causal_attention, METH_FASTCALL, "causal_attention(qkv, batch, rows, heads, kv_heads, head_dim)"},
    {"ter_spmm", (PyCFunction)(void (*)(void))ter_spmm, METH_FASTCALL,
     "ter_spmm(X, row_idx, col_off, tile_idx, batch, rows, columns, inners, uniformed, padded, scale, out, tile_k, prepare)"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", "per-call path of ternaryllm_b200 (see csrc/binding.cpp)", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding(void) { return PyModule_Create(&module); }
