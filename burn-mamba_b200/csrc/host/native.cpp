// Host path of the tensor-level calls (ops.py) and of the block mirrors: argument checks, output allocation, the C
// argument structs of include/bm_b200.h and the launches on torch's current stream, as one CPython extension.
//
// Why it is native: a call of the library used to cost 15-40 us of interpreter time (shape tuples, a ctypes struct
// filled field by field, two or three torch.empty calls), several times the device time of every decode-size kernel.
// The same work takes 2-4 us here.  torch stays what it was: device memory, streams and the library GEMMs.
//
// Every function takes its arguments by position (the Python wrappers own names, defaults and documentation) and
// raises what the wrappers' documentation promises: ValueError for a tensor that does not fit, BmError for a status
// the library returns.  Everything that may block (launches into a full queue, allocations, synchronisation) runs without the
// GIL, like torch's own operators; what is shared between calls is guarded by its own locks.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <optional>
#include <string>
#include <utility>
#include <vector>

#include "decode.h"
#include "mamba3.h"
#include "sizes.h"

using at::Tensor;

namespace {

// ---- the library's entry points, resolved from the .so that _ffi.py loaded ---------------------------------------
#define BM_ENTRY_POINTS(X)                                                                                         \
    X(bm_ssd2_fwd_workspace_bytes) X(bm_ssd2_fwd) X(bm_ssd2_fwd_noalloc) X(bm_workspace_status)                    \
    X(bm_ssd2_bwd_workspace_bytes) X(bm_ssd2_bwd) X(bm_ssd3_bwd_workspace_bytes) X(bm_ssd3_single_bwd)             \
    X(bm_ssd3_double_bwd) X(bm_step2) X(bm_conv_step) X(bm_conv1d_silu_fwd) X(bm_rmsnorm_gated)                    \
    X(bm_mamba3_bc_prep) X(bm_selscan1_fwd) X(bm_selscan1_fwd_workspace_bytes) X(bm_selscan1_fwd_ws) X(bm_step1)   \
    X(bm_ssd3_fwd_workspace_bytes) X(bm_ssd3_single_fwd) X(bm_ssd3_double_fwd) X(bm_angle_cumsum) X(bm_step3)     \
    X(bmx_ssd2_fwd_least_bytes) X(bmx_ssd3_fwd_least_bytes) X(bmx_ssd2_bwd_least_bytes) X(bmx_ssd3_bwd_least_bytes) \
    X(bmx_chain_status) X(bmx_chain_take_status) X(bmx_decode_slices) X(bmx_decode_linear) X(bmx_decode_norm) X(bmx_decode_conv) X(bmx_decode_state)            \
    X(bmx_decode_gated_norm) X(bmx_decode_mixer_sums) X(bmx_decode_mixer)                             \
    X(bmx_m3_coefficients) X(bmx_m3_seed) X(bmx_m3_tail) X(bmx_m3_step_covers) X(bmx_m3_step)
struct Entry {
#define X(n) decltype(&::n) n = nullptr;
    BM_ENTRY_POINTS(X)
#undef X
} L;
PyObject* g_bm_error = nullptr;   // _ffi.BmError

// Failures travel as C++ exceptions, which need no GIL, and become Python's where a function ends (END below).
struct BadValue {
    std::string msg;
};
struct BadStatus {
    int32_t code;
    std::string where;
};
[[noreturn]] void value_error(const std::string& msg) { throw BadValue{msg}; }
void check(int32_t code, const char* where) {
    if (code != BM_OK) throw BadStatus{code, where};
}
[[noreturn]] void rethrow_python() {
    python_error e;
    e.persist();
    throw e;
}
[[noreturn]] void raise(const BadValue& f) {
    PyErr_SetString(PyExc_ValueError, f.msg.c_str());
    rethrow_python();
}
[[noreturn]] void raise(const BadStatus& f) {
    PyObject* exc = PyObject_CallFunction(g_bm_error, "is", (int)f.code, f.where.c_str());   // reads the thread's error string
    if (exc != nullptr) {
        PyErr_SetObject(g_bm_error, exc);
        Py_DECREF(exc);
    }
    rethrow_python();
}

// A scope without the GIL.  Tensors that Python can reach are only read in one.
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    NoGil() = default;
    NoGil(const NoGil&) = delete;
    ~NoGil() { PyEval_RestoreThread(state); }
};
template <typename F>
void launch(const char* where, F f) {
    NoGil scope;
    check(f(), where);
}

// ---- argument access ------------------------------------------------------------------------------------------
const char* dtype_name(at::ScalarType t) { return t == at::kFloat ? "torch.float32" : t == at::kBFloat16 ? "torch.bfloat16" : c10::toString(t); }

std::string shape_str(at::IntArrayRef s) {
    std::string r = "(";
    for (size_t i = 0; i < s.size(); ++i) r += (i ? ", " : "") + std::to_string(s[i]);
    return r + (s.size() == 1 ? ",)" : ")");
}

struct Args {
    PyObject* const* a;
    Py_ssize_t n, i = 0;
    bool exact = true;   // no tensor so far was of a subclass of torch.Tensor
    PyObject* next() {
        if (i >= n) value_error("too few arguments");
        return a[i++];
    }
    int64_t num() {
        const int64_t v = PyLong_AsLongLong(next());
        if (v == -1 && PyErr_Occurred()) rethrow_python();
        return v;
    }
    double real() {
        const double v = PyFloat_AsDouble(next());
        if (v == -1.0 && PyErr_Occurred()) rethrow_python();
        return v;
    }
    bool flag() { return PyObject_IsTrue(next()) == 1; }
    // tensor argument; nullptr for None when optional
    const Tensor* tensor(const char* name, bool optional = false) {
        PyObject* o = next();
        if (o == Py_None) {
            if (optional) return nullptr;
            value_error(std::string(name) + " is required");
        }
        if (!THPVariable_Check(o)) value_error(std::string(name) + " must be a torch.Tensor");
        exact = exact && THPVariable_CheckExact(o);
        return &THPVariable_Unpack(o);
    }
};

void require_cuda(const Tensor& t, const char* name) {
    if (!t.is_cuda()) value_error(std::string(name) + " must be a CUDA tensor (this library has no CPU path)");
}
// CUDA, contiguous, and (when given) dtype and shape
void chk(const Tensor* t, const char* name, c10::optional<at::ScalarType> dtype = c10::nullopt,
         c10::optional<at::IntArrayRef> shape = c10::nullopt) {
    if (t == nullptr) return;
    require_cuda(*t, name);
    if (!t->is_contiguous()) value_error(std::string(name) + " must be contiguous");
    if (dtype && t->scalar_type() != *dtype)
        value_error(std::string(name) + " must be " + dtype_name(*dtype) + ", got " + dtype_name(t->scalar_type()));
    if (shape && t->sizes() != *shape)
        value_error(std::string(name) + " must have shape " + shape_str(*shape) + ", got " + shape_str(t->sizes()));
}
void rank(const Tensor& t, int64_t r, const char* name) {
    if (t.dim() != r) value_error(std::string(name) + " must have " + std::to_string(r) + " axes, got shape " + shape_str(t.sizes()));
}
int32_t dt_code(at::ScalarType t) {
    if (t == at::kFloat) return BM_DTYPE_F32;
    if (t == at::kBFloat16) return BM_DTYPE_BF16;
    value_error(std::string("unsupported activation dtype ") + dtype_name(t));
}
const float* fptr(const Tensor* t) { return t == nullptr ? nullptr : static_cast<const float*>(t->data_ptr()); }
float* fptr(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
const void* vptr(const Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }

Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const Tensor& like) {
    return at::detail::empty_cuda(size, dtype, like.device(), c10::nullopt);
}
void* stream() { return static_cast<void*>(c10::cuda::getCurrentCUDAStream().stream()); }

// Grow-only scratch per (device, stream): the C ABI never allocates.  A buffer belongs to its stream, so launches that
// share it are ordered; there are at most as many entries as streams the program runs the library on.  `m` is held while a
// call's launches go out: the kernels of two threads' calls on one stream would otherwise use the buffer in turns.
struct Workspace {
    std::mutex m;
    Tensor t;
};
std::mutex g_ws_mutex;
std::map<std::pair<int, void*>, Workspace> g_ws;   // entries are never removed
Workspace* find_workspace(int device, bool create) {
    const std::pair<int, void*> key{device, stream()};
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    if (create) return &g_ws[key];
    const auto it = g_ws.find(key);
    return it == g_ws.end() ? nullptr : &it->second;
}
// f(workspace, bytes): one call of the library with a workspace of at least `nbytes`, or of at least `least` where the device
// has no memory for that; with `status_where`, its device status as well (synchronises).
template <typename F>
void with_workspace(size_t nbytes, size_t least, const Tensor& like, const char* where, const char* status_where, F f) {   // without the GIL
    Workspace& w = *find_workspace(like.get_device(), true);
    std::lock_guard<std::mutex> lock(w.m);
    if (!w.t.defined() || (size_t)w.t.numel() < nbytes) {
        try {
            w.t = empty({(int64_t)std::max<size_t>(nbytes, 256)}, at::kByte, like);
        } catch (const c10::OutOfMemoryError&) {
            if (least >= nbytes) throw;
            if (!w.t.defined() || (size_t)w.t.numel() < least) {
                w.t = Tensor();
                w.t = empty({(int64_t)std::max<size_t>(least, 256)}, at::kByte, like);
            }
        }
        w.t.narrow(0, 0, 256).zero_();   // the status word, which not every call writes
    }
    check(f(w.t.data_ptr(), (size_t)w.t.numel()), where);
    if (status_where != nullptr) check(L.bm_workspace_status(w.t.data_ptr(), stream()), status_where);
}
template <typename F>
void launch_ws(size_t nbytes, size_t least, const Tensor& like, const char* where, const char* status_where, F f) {
    NoGil scope;
    with_workspace(nbytes, least, like, where, status_where, f);
}

int32_t* chain_status(int device) {
    int32_t* w = L.bmx_chain_status(device);
    if (w == nullptr) check(BM_ERR_CUDA, "status word of the decode steps");
    return w;
}

PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* none() { Py_RETURN_NONE; }
PyObject* tuple(std::initializer_list<PyObject*> items) {
    PyObject* t = PyTuple_New((Py_ssize_t)items.size());
    Py_ssize_t i = 0;
    for (PyObject* o : items) PyTuple_SET_ITEM(t, i++, o);
    return t;
}
void put(PyObject* dict, const char* key, PyObject* value) {
    PyDict_SetItemString(dict, key, value);
    Py_DECREF(value);
}

// (pointer, row stride) of a tensor whose last axis is contiguous and whose leading axes collapse into rows of one
// stride: dense, or a column slice of a wider row.  Rows that do not start 16-byte aligned are copied (into `keep`;
// the copy is stream-ordered, so it may be released as soon as the launch is enqueued).
const void* rows(const Tensor& t, const char* name, int64_t* stride, Tensor* keep) {
    const int64_t d = t.dim();
    if (t.stride(-1) != 1) value_error(std::string(name) + ": last axis must be contiguous");
    const Tensor* src = &t;
    *stride = d >= 2 ? t.stride(-2) : t.size(-1);
    if ((*stride * (int64_t)t.element_size()) % 16 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) {
        NoGil scope;
        *keep = t.contiguous();
        if (keep->data_ptr() == t.data_ptr()) *keep = t.clone();   // contiguous, yet its base is not aligned
        src = keep;
        *stride = t.size(-1);
    }
    for (int64_t k = 0; k + 2 < d; ++k)
        if (src->stride(k) != src->stride(k + 1) * src->size(k + 1))
            value_error(std::string(name) + ": leading axes must collapse into rows of one stride");
    return src->data_ptr();
}

#define FN(name) PyObject* name(PyObject*, PyObject* const* argv, Py_ssize_t nargs)
#define BEGIN        \
    HANDLE_TH_ERRORS \
    try {            \
        Args A{argv, nargs};
#define END                       \
    }                             \
    catch (const BadValue& f) {   \
        raise(f);                 \
    }                             \
    catch (const BadStatus& f) {  \
        raise(f);                 \
    }                             \
    END_HANDLE_TH_ERRORS

// ---- Mamba-2 SSD -----------------------------------------------------------------------------------------------
// x, dt, a, b, c, d, h0, dt_bias, z, chunk_len, path, dt_min, dt_max, return_states, check_status, reserved, noalloc
FN(ssd2_fwd) {
    BEGIN
    const Tensor &x = *A.tensor("x"), *dt = A.tensor("dt"), *a = A.tensor("a"), &b = *A.tensor("b"), *c = A.tensor("c");
    const Tensor *d = A.tensor("d", true), *h0 = A.tensor("h0", true), *dt_bias = A.tensor("dt_bias", true), *z = A.tensor("z", true);
    bm_ssd2_fwd_args g;
    memset(&g, 0, sizeof g);
    g.chunk_len = (int32_t)A.num(), g.path = (int32_t)A.num();
    g.dt_min = (float)A.real(), g.dt_max = (float)A.real();
    const bool want_states = A.flag(), check_status = A.flag();
    g.reserved = (int32_t)A.num();
    const bool noalloc = A.flag();
    rank(x, 4, "x"), rank(b, 4, "b");
    const int64_t B = x.size(0), S = x.size(1), H = x.size(2), P = x.size(3), G = b.size(2), R = b.size(3);
    const auto act = x.scalar_type();
    g.dtype = dt_code(act);
    chk(&x, "x"), chk(dt, "dt", at::kFloat, at::IntArrayRef{B, S, H}), chk(a, "a", at::kFloat, at::IntArrayRef{H});
    chk(&b, "b", act, at::IntArrayRef{B, S, G, R}), chk(c, "c", act, at::IntArrayRef{B, S, G, R});
    chk(d, "d", at::kFloat, at::IntArrayRef{H}), chk(h0, "h0", at::kFloat, at::IntArrayRef{B, H, P, R});
    chk(dt_bias, "dt_bias", at::kFloat, at::IntArrayRef{H}), chk(z, "z", act, x.sizes());
    Tensor y = empty(x.sizes(), act, x), hf = empty({B, H, P, R}, at::kFloat, x), states;
    const int64_t q = std::max<int64_t>(g.chunk_len, 1);
    if (want_states) states = empty({B, (S + q - 1) / q, H, P, R}, at::kFloat, x);
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.nheads = (int32_t)H, g.headdim = (int32_t)P, g.state_rank = (int32_t)R;
    g.ngroups = (int32_t)G;
    g.x = x.data_ptr(), g.dt = fptr(dt), g.a = fptr(a), g.b = b.data_ptr(), g.c = vptr(c), g.d = fptr(d), g.h0 = fptr(h0);
    g.dt_bias = fptr(dt_bias), g.z = vptr(z), g.y = y.data_ptr(), g.h_final = fptr(hf);
    g.chunk_states = want_states ? fptr(states) : nullptr;
    if (noalloc) {
        launch("bm_ssd2_fwd_noalloc", [&] { return L.bm_ssd2_fwd_noalloc(&g, stream()); });
    } else {
        launch_ws(L.bm_ssd2_fwd_workspace_bytes(&g), L.bmx_ssd2_fwd_least_bytes(&g), x, "bm_ssd2_fwd", check_status ? "bm_ssd2_fwd (device status)" : nullptr,
                  [&](void* ws, size_t n) { return L.bm_ssd2_fwd(&g, ws, n, stream()); });
    }
    if (want_states) return tuple({wrap(y), wrap(hf), wrap(states)});
    return tuple({wrap(y), wrap(hf)});
    END
}

// x, dt, a, b, c, d, h0, dy, dh_final, chunk_len, path, check_status
FN(ssd2_bwd) {
    BEGIN
    const Tensor &x = *A.tensor("x"), *dt = A.tensor("dt"), *a = A.tensor("a"), &b = *A.tensor("b"), *c = A.tensor("c");
    const Tensor *d = A.tensor("d", true), *h0 = A.tensor("h0", true), *dy = A.tensor("dy"), *dhf = A.tensor("dh_final", true);
    bm_ssd2_bwd_args g;
    memset(&g, 0, sizeof g);
    g.chunk_len = (int32_t)A.num(), g.path = (int32_t)A.num();
    const bool check_status = A.flag();
    rank(x, 4, "x"), rank(b, 4, "b");
    const int64_t B = x.size(0), S = x.size(1), H = x.size(2), P = x.size(3), G = b.size(2), R = b.size(3);
    const auto act = x.scalar_type();
    g.dtype = dt_code(act);
    chk(&x, "x"), chk(dt, "dt", at::kFloat, at::IntArrayRef{B, S, H}), chk(a, "a", at::kFloat, at::IntArrayRef{H});
    chk(&b, "b", act, at::IntArrayRef{B, S, G, R}), chk(c, "c", act, at::IntArrayRef{B, S, G, R}), chk(dy, "dy", act, x.sizes());
    chk(d, "d", at::kFloat, at::IntArrayRef{H}), chk(h0, "h0", at::kFloat, at::IntArrayRef{B, H, P, R});
    chk(dhf, "dh_final", at::kFloat, at::IntArrayRef{B, H, P, R});
    Tensor dx = empty(x.sizes(), at::kFloat, x), ddt = empty({B, S, H}, at::kFloat, x), da = empty({H}, at::kFloat, x);
    Tensor db = empty(b.sizes(), at::kFloat, x), dc = empty(b.sizes(), at::kFloat, x), dh0 = empty({B, H, P, R}, at::kFloat, x), dd;
    if (d != nullptr) dd = empty({H}, at::kFloat, x);
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.nheads = (int32_t)H, g.headdim = (int32_t)P, g.state_rank = (int32_t)R;
    g.ngroups = (int32_t)G;
    g.x = x.data_ptr(), g.dt = fptr(dt), g.a = fptr(a), g.b = b.data_ptr(), g.c = vptr(c), g.d = fptr(d), g.h0 = fptr(h0);
    g.dy = vptr(dy), g.dh_final = fptr(dhf), g.dx = fptr(dx), g.ddt = fptr(ddt), g.da = fptr(da), g.db = fptr(db), g.dc = fptr(dc);
    g.dd = d == nullptr ? nullptr : fptr(dd), g.dh0 = fptr(dh0);
    launch_ws(L.bm_ssd2_bwd_workspace_bytes(&g), L.bmx_ssd2_bwd_least_bytes(&g), x, "bm_ssd2_bwd", check_status ? "bm_workspace_status" : nullptr,
              [&](void* ws, size_t n) { return L.bm_ssd2_bwd(&g, ws, n, stream()); });
    PyObject* out = PyDict_New();
    put(out, "dx", wrap(dx)), put(out, "ddt", wrap(ddt)), put(out, "da", wrap(da)), put(out, "db", wrap(db)), put(out, "dc", wrap(dc));
    put(out, "dd", d == nullptr ? none() : wrap(dd)), put(out, "dh0", wrap(dh0));
    return out;
    END
}

// state, x, dt, a, b, c, d, dt_bias, z, dt_min, dt_max
FN(step2) {
    BEGIN
    const Tensor &st = *A.tensor("state"), &x = *A.tensor("x"), *dt = A.tensor("dt"), *a = A.tensor("a"), &b = *A.tensor("b"), *c = A.tensor("c");
    const Tensor *d = A.tensor("d", true), *dt_bias = A.tensor("dt_bias", true), *z = A.tensor("z", true);
    bm_step2_args g;
    memset(&g, 0, sizeof g);
    g.dt_min = (float)A.real(), g.dt_max = (float)A.real();
    rank(st, 4, "state"), rank(b, 3, "b");
    const int64_t B = st.size(0), H = st.size(1), P = st.size(2), R = st.size(3), G = b.size(1);
    const auto act = x.scalar_type();
    g.dtype = dt_code(act);
    chk(&st, "state", at::kFloat), chk(&x, "x", act, at::IntArrayRef{B, H, P}), chk(dt, "dt", at::kFloat, at::IntArrayRef{B, H});
    chk(a, "a", at::kFloat, at::IntArrayRef{H}), chk(&b, "b", act, at::IntArrayRef{B, G, R}), chk(c, "c", act, at::IntArrayRef{B, G, R});
    chk(d, "d", at::kFloat, at::IntArrayRef{H}), chk(dt_bias, "dt_bias", at::kFloat, at::IntArrayRef{H}), chk(z, "z", act, at::IntArrayRef{B, H, P});
    Tensor y = empty(x.sizes(), act, x);
    g.batch = (int32_t)B, g.nheads = (int32_t)H, g.headdim = (int32_t)P, g.state_rank = (int32_t)R, g.ngroups = (int32_t)G;
    g.state = fptr(st), g.x = x.data_ptr(), g.dt = fptr(dt), g.a = fptr(a), g.b = b.data_ptr(), g.c = vptr(c), g.d = fptr(d);
    g.dt_bias = fptr(dt_bias), g.z = vptr(z), g.y = y.data_ptr();
    launch("bm_step2", [&] { return L.bm_step2(&g, stream()); });
    return wrap(y);
    END
}

// ---- conv, norm --------------------------------------------------------------------------------------------------
struct Splits {
    bool on;
    int64_t sx, sbc;
};
Splits read_splits(Args& A, int64_t v) {   // three integers; the first is negative for "one tensor"
    const int64_t sx = A.num(), sbc = A.num(), sbc2 = A.num();
    if (sx < 0) return {false, 0, 0};
    if (sbc != sbc2 || sx + 2 * sbc != v) value_error("splits must be (split_x, split_bc, split_bc) summing to the channel count");
    return {true, sx, sbc};
}

// window, xin, weight, bias, splits...
FN(conv_step) {
    BEGIN
    const Tensor &win = *A.tensor("window"), &xin = *A.tensor("xin"), *w = A.tensor("weight"), *bias = A.tensor("bias", true);
    rank(win, 3, "window");
    const int64_t B = win.size(0), V = win.size(1), K = win.size(2);
    chk(&win, "window", at::kFloat);
    if (!xin.is_cuda() || xin.dim() != 2 || xin.size(0) != B || xin.size(1) != V || xin.stride(1) != 1)
        value_error("xin must be a CUDA tensor [b, v] with a contiguous last axis");
    chk(w, "weight", at::kFloat, at::IntArrayRef{V, K}), chk(bias, "bias", at::kFloat, at::IntArrayRef{V});
    const auto act = xin.scalar_type();
    bm_conv_step_args g;
    memset(&g, 0, sizeof g);
    g.dtype = dt_code(act);
    const Splits s = read_splits(A, V);
    Tensor o, ob, oc;
    if (s.on) {
        o = empty({B, s.sx}, act, xin), ob = empty({B, s.sbc}, act, xin), oc = empty({B, s.sbc}, act, xin);
        g.out_b = ob.data_ptr(), g.out_c = oc.data_ptr();
    } else {
        o = empty({B, V}, act, xin);
    }
    g.batch = (int32_t)B, g.channels = (int32_t)V, g.kernel = (int32_t)K, g.window = fptr(win), g.xin = xin.data_ptr();
    g.weight = fptr(w), g.bias = fptr(bias), g.out = o.data_ptr(), g.xin_stride = (int32_t)xin.stride(0);
    g.split_x = (int32_t)s.sx, g.split_bc = (int32_t)s.sbc;
    launch("bm_conv_step", [&] { return L.bm_conv_step(&g, stream()); });
    return s.on ? tuple({wrap(o), wrap(ob), wrap(oc)}) : wrap(o);
    END
}

// xbc, weight, bias, window, want_window, splits...
FN(conv1d_silu_fwd) {
    BEGIN
    const Tensor &xbc = *A.tensor("xbc"), &w = *A.tensor("weight"), *bias = A.tensor("bias", true), *win = A.tensor("window", true);
    const bool want_window = A.flag();
    rank(xbc, 3, "xbc"), rank(w, 2, "weight");
    const int64_t B = xbc.size(0), S = xbc.size(1), V = xbc.size(2), K = w.size(1);
    const auto act = xbc.scalar_type();
    require_cuda(xbc, "xbc");
    bm_conv1d_silu_args g;
    memset(&g, 0, sizeof g);
    g.dtype = dt_code(act);
    int64_t stride;
    Tensor keep;
    g.xin = rows(xbc, "xbc", &stride, &keep);
    chk(&w, "weight", at::kFloat, at::IntArrayRef{V, K}), chk(bias, "bias", at::kFloat, at::IntArrayRef{V});
    chk(win, "window", at::kFloat, at::IntArrayRef{B, V, K});
    const Splits s = read_splits(A, V);
    Tensor o, ob, oc, nw;
    if (want_window) nw = empty({B, V, K}, at::kFloat, xbc);
    if (s.on) {
        o = empty({B, S, s.sx}, act, xbc), ob = empty({B, S, s.sbc}, act, xbc), oc = empty({B, S, s.sbc}, act, xbc);
        g.out_b = ob.data_ptr(), g.out_c = oc.data_ptr();
    } else {
        o = empty({B, S, V}, act, xbc);
    }
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.channels = (int32_t)V, g.kernel = (int32_t)K, g.xin_stride = (int32_t)stride;
    g.split_x = (int32_t)s.sx, g.split_bc = (int32_t)s.sbc, g.weight = fptr(w), g.bias = fptr(bias), g.window = fptr(win);
    g.new_window = want_window ? fptr(nw) : nullptr, g.out_x = o.data_ptr();
    launch("bm_conv1d_silu_fwd", [&] { return L.bm_conv1d_silu_fwd(&g, stream()); });
    PyObject* outs = s.on ? tuple({wrap(o), wrap(ob), wrap(oc)}) : wrap(o);
    return tuple({outs, want_window ? wrap(nw) : none()});
    END
}

// x, z, gamma, norm_before_gate, eps
FN(rmsnorm_gated) {
    BEGIN
    const Tensor &x = *A.tensor("x"), *z = A.tensor("z", true), *gamma = A.tensor("gamma");
    bm_rmsnorm_gated_args g;
    memset(&g, 0, sizeof g);
    g.norm_before_gate = A.flag(), g.eps = (float)A.real();
    const int64_t d = x.size(-1);
    if (d < 1) value_error("x must have at least one column");
    const auto act = x.scalar_type();
    require_cuda(x, "x");
    g.dtype = dt_code(act);
    int64_t xs = 0, zs = 0;
    Tensor keepx, keepz;
    g.x = rows(x, "x", &xs, &keepx);
    if (z != nullptr) g.z = rows(*z, "z", &zs, &keepz);
    chk(gamma, "gamma", act, at::IntArrayRef{d});
    Tensor out = empty(x.sizes(), act, x);
    g.rows = (int32_t)(out.numel() / d), g.width = (int32_t)d, g.x_stride = (int32_t)xs, g.z_stride = (int32_t)zs;
    g.gamma = vptr(gamma), g.out = out.data_ptr();
    launch("bm_rmsnorm_gated", [&] { return L.bm_rmsnorm_gated(&g, stream()); });
    return wrap(out);
    END
}

// ---- Mamba-1 -------------------------------------------------------------------------------------------------------
// u, delta, a, b, c, d, z, h0, delta_bias, delta_softplus, serial
FN(selscan1_fwd) {
    BEGIN
    const Tensor &u = *A.tensor("u"), *delta = A.tensor("delta"), &a = *A.tensor("a"), *b = A.tensor("b"), *c = A.tensor("c");
    const Tensor *d = A.tensor("d", true), *z = A.tensor("z", true), *h0 = A.tensor("h0", true), *db = A.tensor("delta_bias", true);
    bm_selscan1_args g;
    memset(&g, 0, sizeof g);
    g.delta_softplus = A.flag();
    const bool serial = A.flag();
    rank(u, 3, "u"), rank(a, 2, "a");
    const int64_t B = u.size(0), S = u.size(1), I = u.size(2), R = a.size(1);
    const auto act = u.scalar_type();
    g.dtype = dt_code(act);
    chk(&u, "u"), chk(delta, "delta", act, at::IntArrayRef{B, S, I}), chk(&a, "a", at::kFloat, at::IntArrayRef{I, R});
    chk(b, "b", act, at::IntArrayRef{B, S, R}), chk(c, "c", act, at::IntArrayRef{B, S, R}), chk(d, "d", at::kFloat, at::IntArrayRef{I});
    chk(z, "z", act, at::IntArrayRef{B, S, I}), chk(h0, "h0", at::kFloat, at::IntArrayRef{B, I, R}), chk(db, "delta_bias", at::kFloat, at::IntArrayRef{I});
    Tensor y = empty(u.sizes(), act, u), hf = empty({B, I, R}, at::kFloat, u);
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.d_inner = (int32_t)I, g.state_rank = (int32_t)R;
    g.u = u.data_ptr(), g.delta = vptr(delta), g.a = fptr(&a), g.b = vptr(b), g.c = vptr(c), g.d = fptr(d), g.delta_bias = fptr(db);
    g.z = vptr(z), g.h0 = fptr(h0), g.y = y.data_ptr(), g.h_final = fptr(hf);
    if (serial) {
        launch("bm_selscan1_fwd", [&] { return L.bm_selscan1_fwd(&g, stream()); });
    } else {
        const size_t need = L.bm_selscan1_fwd_workspace_bytes(&g);
        launch_ws(need, need, u, "bm_selscan1_fwd_ws", nullptr,
                  [&](void* ws, size_t n) { return L.bm_selscan1_fwd_ws(&g, ws, n, stream()); });
    }
    return tuple({wrap(y), wrap(hf)});
    END
}

// state, u, delta, a, b, c, d, z, delta_bias, delta_softplus
FN(step1) {
    BEGIN
    const Tensor &st = *A.tensor("state"), &u = *A.tensor("u"), *delta = A.tensor("delta"), *a = A.tensor("a"), *b = A.tensor("b"), *c = A.tensor("c");
    const Tensor *d = A.tensor("d", true), *z = A.tensor("z", true), *db = A.tensor("delta_bias", true);
    bm_step1_args g;
    memset(&g, 0, sizeof g);
    g.delta_softplus = A.flag();
    rank(st, 3, "state");
    const int64_t B = st.size(0), I = st.size(1), R = st.size(2);
    const auto act = u.scalar_type();
    g.dtype = dt_code(act);
    chk(&st, "state", at::kFloat), chk(&u, "u", act, at::IntArrayRef{B, I}), chk(delta, "delta", act, at::IntArrayRef{B, I});
    chk(a, "a", at::kFloat, at::IntArrayRef{I, R}), chk(b, "b", act, at::IntArrayRef{B, R}), chk(c, "c", act, at::IntArrayRef{B, R});
    chk(d, "d", at::kFloat, at::IntArrayRef{I}), chk(z, "z", act, at::IntArrayRef{B, I}), chk(db, "delta_bias", at::kFloat, at::IntArrayRef{I});
    Tensor y = empty(u.sizes(), act, u);
    g.batch = (int32_t)B, g.d_inner = (int32_t)I, g.state_rank = (int32_t)R;
    g.state = fptr(st), g.u = u.data_ptr(), g.delta = vptr(delta), g.a = fptr(a), g.b = vptr(b), g.c = vptr(c), g.d = fptr(d);
    g.delta_bias = fptr(db), g.z = vptr(z), g.y = y.data_ptr();
    launch("bm_step1", [&] { return L.bm_step1(&g, stream()); });
    return wrap(y);
    END
}

// ---- Mamba-3 -------------------------------------------------------------------------------------------------------
// b_raw, c_raw, b_gamma, c_gamma, b_bias, c_bias, angles, rope_dim (-1: state_rank), pairwise (-1: mimo_rank == 1), ngroups, eps
FN(mamba3_bc_prep) {
    BEGIN
    const Tensor &br = *A.tensor("b_raw"), &cr = *A.tensor("c_raw"), *bg = A.tensor("b_gamma"), *cg = A.tensor("c_gamma");
    const Tensor &bb = *A.tensor("b_bias"), *cb = A.tensor("c_bias"), *ang = A.tensor("angles", true);
    int64_t rope = A.num(), pairwise = A.num();
    const int64_t G = A.num();
    const double eps = A.real();
    rank(br, 3, "b_raw"), rank(bb, 3, "b_bias");
    const int64_t B = br.size(0), S = br.size(1), mgr = br.size(2), H = bb.size(0), M = bb.size(1), R = bb.size(2);
    const auto act = br.scalar_type();
    require_cuda(br, "b_raw");
    if (mgr != M * G * R || cr.sizes() != br.sizes()) value_error("raw rows must hold m * g * r entries");
    if (rope < 0) rope = R;
    if (pairwise < 0) pairwise = M == 1;
    bm_mamba3_bc_prep_args g;
    memset(&g, 0, sizeof g);
    g.dtype = dt_code(act);
    int64_t bs, cs;
    Tensor keepb, keepc;
    g.b_raw = rows(br, "b_raw", &bs, &keepb), g.c_raw = rows(cr, "c_raw", &cs, &keepc);
    if (bs != cs) value_error("b_raw and c_raw must have the same row stride");
    chk(bg, "b_gamma", at::kFloat, at::IntArrayRef{R}), chk(cg, "c_gamma", at::kFloat, at::IntArrayRef{R});
    chk(&bb, "b_bias", at::kFloat, at::IntArrayRef{H, M, R}), chk(cb, "c_bias", at::kFloat, at::IntArrayRef{H, M, R});
    chk(ang, "angles", at::kFloat, at::IntArrayRef{B, S, H, std::max<int64_t>(rope / 2, 0)});
    Tensor ob = empty({B, S, M, H, R}, act, br), oc = empty({B, S, M, H, R}, act, br);
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.mimo_rank = (int32_t)M, g.ngroups = (int32_t)G, g.nheads = (int32_t)H;
    g.state_rank = (int32_t)R, g.raw_stride = (int32_t)bs, g.rope_dim = (int32_t)rope, g.pairwise = (int32_t)pairwise, g.eps = (float)eps;
    g.b_gamma = fptr(bg), g.c_gamma = fptr(cg), g.b_bias = fptr(&bb), g.c_bias = fptr(cb), g.angles = fptr(ang);
    g.b_out = ob.data_ptr(), g.c_out = oc.data_ptr();
    launch("bm_mamba3_bc_prep", [&] { return L.bm_mamba3_bc_prep(&g, stream()); });
    return tuple({wrap(ob), wrap(oc)});
    END
}

// single, v, da, b, c, gamma, scale, h0, angles, chunk_len, rope_dim, path, check_status
FN(ssd3_fwd) {
    BEGIN
    const bool single = A.flag();
    const Tensor &v = *A.tensor("v"), *da = A.tensor("da"), &b = *A.tensor("b"), *c = A.tensor("c"), *gamma = A.tensor("gamma", true);
    const Tensor *scale = A.tensor("scale", true), *h0 = A.tensor("h0", true), *ang = A.tensor("angles", true);
    bm_ssd3_fwd_args g;
    memset(&g, 0, sizeof g);
    g.chunk_len = (int32_t)A.num(), g.rope_dim = (int32_t)A.num(), g.path = (int32_t)A.num();
    const bool check_status = A.flag();
    rank(v, 5, "v"), rank(b, 5, "b");
    const int64_t B = v.size(0), S = v.size(1), M = v.size(2), H = v.size(3), P = v.size(4), R = b.size(4);
    const auto act = v.scalar_type();
    g.dtype = dt_code(act);
    chk(&v, "v"), chk(da, "da", at::kFloat, at::IntArrayRef{B, S, H}), chk(&b, "b", act, at::IntArrayRef{B, S, M, H, R});
    chk(c, "c", act, at::IntArrayRef{B, S, M, H, R}), chk(gamma, "gamma", at::kFloat, at::IntArrayRef{B, S, H});
    chk(scale, "scale", at::kFloat, at::IntArrayRef{B, S, H}), chk(h0, "h0", at::kFloat, at::IntArrayRef{B, H, P, R});
    chk(ang, "angles", at::kFloat, at::IntArrayRef{B, S, H, std::max<int64_t>(g.rope_dim / 2, 1)});
    Tensor y = empty(v.sizes(), act, v), hf = empty({B, H, P, R}, at::kFloat, v);
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.nheads = (int32_t)H, g.headdim = (int32_t)P, g.state_rank = (int32_t)R;
    g.mimo_rank = (int32_t)M;
    g.v = v.data_ptr(), g.da = fptr(da), g.b = b.data_ptr(), g.c = vptr(c), g.gamma = fptr(gamma), g.scale = fptr(scale);
    g.h0 = fptr(h0), g.angles = fptr(ang), g.y = y.data_ptr(), g.h_final = fptr(hf);
    const std::string name = single ? "bm_ssd3_single_fwd" : "bm_ssd3_double_fwd", status_name = name + " (device status)";
    launch_ws(L.bm_ssd3_fwd_workspace_bytes(&g), L.bmx_ssd3_fwd_least_bytes(&g), v, name.c_str(), check_status ? status_name.c_str() : nullptr,
              [&](void* ws, size_t n) { return (single ? L.bm_ssd3_single_fwd : L.bm_ssd3_double_fwd)(&g, ws, n, stream()); });
    return tuple({wrap(y), wrap(hf)});
    END
}

// single, v, da, b, c, gamma, scale, h0, dy, dh_final, chunk_len, path, check_status
FN(ssd3_bwd) {
    BEGIN
    const bool single = A.flag();
    const Tensor &v = *A.tensor("v"), *da = A.tensor("da"), &b = *A.tensor("b"), *c = A.tensor("c"), *gamma = A.tensor("gamma", !single);
    const Tensor *scale = A.tensor("scale", !single), *h0 = A.tensor("h0", true), *dy = A.tensor("dy"), *dhf = A.tensor("dh_final", true);
    bm_ssd3_bwd_args g;
    memset(&g, 0, sizeof g);
    g.chunk_len = (int32_t)A.num(), g.path = (int32_t)A.num();
    const bool check_status = A.flag();
    rank(v, 5, "v"), rank(b, 5, "b");
    const int64_t B = v.size(0), S = v.size(1), M = v.size(2), H = v.size(3), P = v.size(4), R = b.size(4);
    const auto act = v.scalar_type();
    g.dtype = dt_code(act);
    chk(&v, "v"), chk(da, "da", at::kFloat, at::IntArrayRef{B, S, H}), chk(&b, "b", act, at::IntArrayRef{B, S, M, H, R});
    chk(c, "c", act, at::IntArrayRef{B, S, M, H, R}), chk(dy, "dy", act, v.sizes()), chk(h0, "h0", at::kFloat, at::IntArrayRef{B, H, P, R});
    chk(dhf, "dh_final", at::kFloat, at::IntArrayRef{B, H, P, R});
    Tensor dv = empty(v.sizes(), at::kFloat, v), dda = empty({B, S, H}, at::kFloat, v), db = empty(b.sizes(), at::kFloat, v);
    Tensor dc = empty(b.sizes(), at::kFloat, v), dh0 = empty({B, H, P, R}, at::kFloat, v), dgamma, dscale;
    if (single) {
        chk(gamma, "gamma", at::kFloat, at::IntArrayRef{B, S, H}), chk(scale, "scale", at::kFloat, at::IntArrayRef{B, S, H});
        dgamma = empty({B, S, H}, at::kFloat, v), dscale = empty({B, S, H}, at::kFloat, v);
        g.gamma = fptr(gamma), g.scale = fptr(scale), g.dgamma = fptr(dgamma), g.dscale = fptr(dscale);
    }
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.nheads = (int32_t)H, g.headdim = (int32_t)P, g.state_rank = (int32_t)R;
    g.mimo_rank = (int32_t)M;
    g.v = v.data_ptr(), g.da = fptr(da), g.b = b.data_ptr(), g.c = vptr(c), g.h0 = fptr(h0), g.dy = vptr(dy), g.dh_final = fptr(dhf);
    g.dv = fptr(dv), g.dda = fptr(dda), g.db = fptr(db), g.dc = fptr(dc), g.dh0 = fptr(dh0);
    launch_ws(L.bm_ssd3_bwd_workspace_bytes(&g), L.bmx_ssd3_bwd_least_bytes(&g), v, "bm_ssd3_bwd", check_status ? "bm_workspace_status" : nullptr,
              [&](void* ws, size_t n) { return (single ? L.bm_ssd3_single_bwd : L.bm_ssd3_double_bwd)(&g, ws, n, stream()); });
    PyObject* out = PyDict_New();
    put(out, "dv", wrap(dv)), put(out, "dda", wrap(dda)), put(out, "db", wrap(db)), put(out, "dc", wrap(dc)), put(out, "dh0", wrap(dh0));
    if (single) put(out, "dgamma", wrap(dgamma)), put(out, "dscale", wrap(dscale));
    return out;
    END
}

// rot, dt, prev, range
FN(angle_cumsum) {
    BEGIN
    const Tensor &rot = *A.tensor("rot"), &dt = *A.tensor("dt"), *prev = A.tensor("prev", true);
    bm_angle_cumsum_args g;
    memset(&g, 0, sizeof g);
    g.range = (float)A.real();
    rank(rot, 3, "rot"), rank(dt, 3, "dt");
    const int64_t B = rot.size(0), S = rot.size(1), NA = rot.size(2), H = dt.size(2);
    chk(&rot, "rot", at::kFloat), chk(&dt, "dt", at::kFloat, at::IntArrayRef{B, S, H}), chk(prev, "prev", at::kFloat, at::IntArrayRef{B, H, NA});
    Tensor theta = empty({B, S, H, NA}, at::kFloat, rot), last = empty({B, H, NA}, at::kFloat, rot);
    g.batch = (int32_t)B, g.seqlen = (int32_t)S, g.nheads = (int32_t)H, g.nangles = (int32_t)NA;
    g.rot = fptr(&rot), g.dt = fptr(&dt), g.prev = fptr(prev), g.theta = fptr(theta), g.last = fptr(last);
    launch("bm_angle_cumsum", [&] { return L.bm_angle_cumsum(&g, stream()); });
    return tuple({wrap(theta), wrap(last)});
    END
}

// state, k_state, v_state, angle, x, b, c, rot, dt, alpha, beta, gamma, mimo_x, rope_dim (-1: state_rank), range
FN(step3) {
    BEGIN
    const Tensor &st = *A.tensor("state"), &ks = *A.tensor("k_state"), &vs = *A.tensor("v_state"), &ang = *A.tensor("angle"), *x = A.tensor("x");
    const Tensor &b = *A.tensor("b"), *c = A.tensor("c"), *rot = A.tensor("rot"), *dt = A.tensor("dt"), *al = A.tensor("alpha");
    const Tensor *be = A.tensor("beta"), *ga = A.tensor("gamma"), *mx = A.tensor("mimo_x", true);
    int64_t rope = A.num();
    bm_step3_args g;
    memset(&g, 0, sizeof g);
    g.range = (float)A.real();
    rank(st, 4, "state"), rank(b, 4, "b");
    const int64_t B = st.size(0), H = st.size(1), P = st.size(2), R = st.size(3), M = b.size(1);
    if (rope < 0) rope = R;
    const int64_t NA = std::max<int64_t>(rope / 2, 1);
    const auto f = at::kFloat;
    chk(&st, "state", f), chk(&ks, "k_state", f, at::IntArrayRef{B, M, H, R}), chk(&vs, "v_state", f, at::IntArrayRef{B, H, P});
    chk(&ang, "angle", f, at::IntArrayRef{B, H, NA}), chk(x, "x", f, at::IntArrayRef{B, H, P}), chk(&b, "b", f, at::IntArrayRef{B, M, H, R});
    chk(c, "c", f, at::IntArrayRef{B, M, H, R}), chk(rot, "rot", f, at::IntArrayRef{B, NA}), chk(dt, "dt", f, at::IntArrayRef{B, H});
    chk(al, "alpha", f, at::IntArrayRef{B, H}), chk(be, "beta", f, at::IntArrayRef{B, H}), chk(ga, "gamma", f, at::IntArrayRef{B, H});
    chk(mx, "mimo_x", f, at::IntArrayRef{H, M, P});
    Tensor y = empty({B, M, H, P}, f, st);
    g.batch = (int32_t)B, g.nheads = (int32_t)H, g.headdim = (int32_t)P, g.state_rank = (int32_t)R, g.mimo_rank = (int32_t)M;
    g.rope_dim = (int32_t)rope;
    g.state = fptr(st), g.k_state = fptr(ks), g.v_state = fptr(vs), g.angle = fptr(ang), g.x = fptr(x), g.b = fptr(&b), g.c = fptr(c);
    g.rot = fptr(rot), g.dt = fptr(dt), g.alpha = fptr(al), g.beta = fptr(be), g.gamma = fptr(ga), g.mimo_x = fptr(mx), g.y = fptr(y);
    launch("bm_step3", [&] { return L.bm_step3(&g, stream()); });
    return wrap(y);
    END
}

// ---- fused decode step of Mamba-2 layers (decode.h) -------------------------------------------------------------------
struct M2Layer {
    Tensor w_in, conv_w, conv_b, dt_bias, a, d, gamma, w_out, window, state, norm;   // norm undefined: no layer norm
    int64_t H, P, G, V, DI, N;
    int before_gate;
    float dt_min, dt_max;
};
// A tensor whose values are what lies at its pointer, for any reader.  Not so: tensors that dispatch elsewhere (subclasses
// without storage, batched, functional or sparse tensors; everything while a dispatch mode watches), lazy negations, zeros
// without memory.
bool plain(const Tensor& t) {
    return !at::isTensorSubclassLike(t) && t.layout() == at::kStrided && !t.is_neg() && !t._is_zerotensor() && t.has_storage() && t.data_ptr() != nullptr;
}
// `like`: the activations of the call, on whose device every operand has to be.
bool dense(const Tensor& t, at::ScalarType dt, at::IntArrayRef shape, const Tensor& like) {
    return t.defined() && t.is_cuda() && plain(t) && t.device() == like.device() && t.scalar_type() == dt && t.sizes() == shape && t.is_contiguous() &&
           reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && !(c10::GradMode::is_enabled() && t.requires_grad()) && !t._fw_grad(0).defined();
}
// The chains launch on the current device's stream and read every operand there.
bool elsewhere(const Tensor& t) { return t.get_device() != c10::cuda::current_device(); }
// Under autocast torch picks the type of every product: the native chains take their operands as they are, so such calls
// keep the op-by-op form.
bool autocasting() { return at::autocast::is_autocast_enabled(at::kCUDA); }
// Fills `l` from the tuple (w_in, conv_w, conv_b, dt_bias, a, d, gamma, w_out, window, state, norm | None, nheads, ngroups,
// norm_before_gate, dt_min, dt_max); false when the chain does not cover the layer.
bool read_layer(PyObject* tup, const Tensor& x, M2Layer& l) {
    const int64_t B = x.size(0), DM = x.size(1);
    Tensor* ts[] = {&l.w_in, &l.conv_w, &l.conv_b, &l.dt_bias, &l.a, &l.d, &l.gamma, &l.w_out, &l.window, &l.state, &l.norm};
    if (!PyTuple_Check(tup) || PyTuple_GET_SIZE(tup) != 16) return false;
    for (int i = 0; i < 11; ++i) {
        PyObject* o = PyTuple_GET_ITEM(tup, i);
        if (THPVariable_CheckExact(o)) *ts[i] = THPVariable_Unpack(o);   // a subclass may redefine the products: not the chain's
        else if (o != Py_None || i != 10) return false;
    }
    l.H = PyLong_AsLongLong(PyTuple_GET_ITEM(tup, 11)), l.G = PyLong_AsLongLong(PyTuple_GET_ITEM(tup, 12));
    l.before_gate = PyObject_IsTrue(PyTuple_GET_ITEM(tup, 13));
    l.dt_min = (float)PyFloat_AsDouble(PyTuple_GET_ITEM(tup, 14)), l.dt_max = (float)PyFloat_AsDouble(PyTuple_GET_ITEM(tup, 15));
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    constexpr int64_t R = 128, K = 4;
    const auto bf = at::kBFloat16, f = at::kFloat;
    if (l.state.dim() != 4 || l.H < 1 || l.G < 1 || l.H % l.G) return false;
    l.P = l.state.size(2), l.DI = l.H * l.P, l.V = l.DI + 2 * l.G * R, l.N = l.DI + l.V + l.H;
    if (l.DI % 8 || l.N % 8 || DM % 8 || l.DI > 8192 || DM > 8192) return false;
    return dense(l.w_in, bf, {DM, l.N}, x) && dense(l.w_out, bf, {l.DI, DM}, x) && dense(l.gamma, bf, {l.DI}, x) && dense(l.conv_w, f, {l.V, K}, x) &&
           dense(l.conv_b, f, {l.V}, x) && dense(l.dt_bias, f, {l.H}, x) && dense(l.a, f, {l.H}, x) && dense(l.d, f, {l.H}, x) &&
           dense(l.window, f, {B, l.V, K}, x) && dense(l.state, f, {B, l.H, l.P, R}, x) && (!l.norm.defined() || dense(l.norm, bf, {DM}, x));
}

// layers (list of tuples), x [b, d_model] bf16, residual | None (only without layer norms), eps -> y [b, d_model], or None
// when the chain does not cover the call (the caller then runs the step kernel by kernel).  A wait that ran out in an earlier
// step on the device is raised here; with a fifth argument that is true, one of this step (synchronises).
// With layer norms: x <- x + step(norm(x)) per layer; without: step(x) (+ residual) of the one layer.
FN(m2_decode) {
    BEGIN
    PyObject* list = A.next();
    const Tensor &x = *A.tensor("x"), *residual = A.tensor("residual", true);
    const float eps = (float)A.real();
    const bool check_status = A.i < A.n && A.flag();
    if (!PyList_Check(list) || PyList_GET_SIZE(list) == 0 || x.dim() != 2) return none();
    const int64_t B = x.size(0), DM = x.size(1), n = PyList_GET_SIZE(list);
    if (!A.exact || autocasting() || B < 1 || B > 131070 /* two rows per block of a 65535-wide grid axis */ || !dense(x, at::kBFloat16, {B, DM}, x) || (residual && !dense(*residual, at::kBFloat16, {B, DM}, x))) return none();
    std::vector<M2Layer> ls((size_t)n);
    for (int64_t i = 0; i < n; ++i)
        if (!read_layer(PyList_GET_ITEM(list, i), x, ls[(size_t)i])) return none();
    const bool norms = ls[0].norm.defined();
    for (auto& l : ls)
        if (l.norm.defined() != norms) return none();
    if ((!norms && n != 1) || elsewhere(x)) return none();
    // the chain reads a layer's caches before the kernels of earlier layers have ended: layers that share one run in order
    std::vector<std::pair<uintptr_t, uintptr_t>> spans;
    for (auto& l : ls)
        for (const Tensor* t : {&l.window, &l.state}) {
            const uintptr_t p = reinterpret_cast<uintptr_t>(t->data_ptr());
            spans.emplace_back(p, p + t->nbytes());
        }
    std::sort(spans.begin(), spans.end());
    for (size_t i = 1; i < spans.size(); ++i)
        if (spans[i].first < spans[i - 1].second) return none();
    // streaming projections up to a batch of 8, library products above
    bool stream_w = true;
    for (auto& l : ls)
        stream_w = stream_w && L.bmx_decode_slices((int32_t)B, (int32_t)DM, (int32_t)l.N) > 0 && L.bmx_decode_slices((int32_t)B, (int32_t)l.DI, (int32_t)DM) > 0;
    // scratch of the whole chain: one allocation, carved; every layer reuses it (stream order)
    int64_t off = 0;
    auto carve = [&](int64_t bytes) {
        const int64_t o = off;
        off += (bytes + 255) / 256 * 256;
        return o;
    };
    int64_t di = 0, gr = 0, nn = 0, p1 = 0, p2 = 0, nss = 0;
    for (auto& l : ls) {
        di = std::max(di, l.DI), gr = std::max(gr, l.G * 128), nn = std::max(nn, l.N);
        if (stream_w) {
            p1 = std::max<int64_t>(p1, L.bmx_decode_slices((int32_t)B, (int32_t)DM, (int32_t)l.N) * l.N);
            nss = std::max<int64_t>(nss, L.bmx_decode_mixer_sums((int32_t)B, (int32_t)l.H, (int32_t)l.P));
            p2 = std::max<int64_t>(p2, L.bmx_decode_slices((int32_t)B, (int32_t)l.DI, (int32_t)DM) * DM);
        }
    }
    const int32_t planes = stream_w ? 2 : 1;
    const int64_t o_norm = carve(planes * B * DM * 2), o_x = carve(B * di * 2), o_b = carve(B * gr * 2), o_c = carve(B * gr * 2), o_y = carve(B * di * 2);
    const int64_t o_g = carve(planes * B * di * 2), o_r0 = carve(B * DM * 4), o_r1 = carve(B * DM * 4);
    const int64_t o_p1 = carve(stream_w ? B * p1 * 4 : B * nn * 2), o_p2 = carve(stream_w ? B * p2 * 4 : 0), o_ss = carve(B * nss * 4);
    Tensor scratch = empty({off}, at::kByte, x), out = empty({B, DM}, at::kBFloat16, x);
    char* base = static_cast<char*>(scratch.data_ptr());
    auto view = [&](int64_t o, int64_t rows, int64_t cols) {
        return at::from_blob(base + o, {rows, cols}, at::TensorOptions().dtype(at::kBFloat16).device(x.device()));
    };
    std::optional<NoGil> scope;   // until the result is wrapped
    scope.emplace();
    int32_t* status = chain_status(x.get_device());
    check(L.bmx_chain_take_status(status), "decode step (an earlier one)");
    void* st = stream();
    const void* xres = norms ? x.data_ptr() : residual ? residual->data_ptr() : nullptr;   // the residual stream
    const float* xres32 = nullptr;
    bmx_rows add{};   // what the last out-projection left, still to be added to the residual stream
    bmx_mixer mix{};
    bool have_add = false, fused = false;   // fused: the last layer ran the fused mixer
    for (int64_t i = 0; i < n; ++i) {
        M2Layer& l = ls[(size_t)i];
        const void* in = x.data_ptr();
        if (norms) {
            // streaming path: x' = xres + add is kept in float32 from the second layer on; library path: the stream lives in `out`
            float* xo32 = have_add ? reinterpret_cast<float*>(base + (i & 1 ? o_r1 : o_r0)) : nullptr;
            void* xo = !stream_w && i == 0 ? out.data_ptr() : nullptr;
            check(L.bmx_decode_norm(xres, xres32, have_add ? &add : nullptr, fused ? &mix : nullptr, l.norm.data_ptr(), eps, xo32, xo, base + o_norm, planes, (int32_t)B,
                                    (int32_t)DM, i == 0, st), "decode step (norm)");
            if (xo) xres = xo;
            if (xo32) xres = nullptr, xres32 = xo32;
            in = base + o_norm;
        }
        bmx_rows proj{};
        proj.ld = l.N;
        if (stream_w) {
            proj.nslice = L.bmx_decode_slices((int32_t)B, (int32_t)DM, (int32_t)l.N);
            proj.slice = B * l.N;
            float* p = reinterpret_cast<float*>(base + o_p1);
            check(L.bmx_decode_linear(in, norms ? planes : 1, l.w_in.data_ptr(), p, (int32_t)B, (int32_t)DM, (int32_t)l.N, proj.nslice, status, !norms, 0, st), "decode step (in-projection)");
            proj.part = p;
        } else {
            Tensor po = view(o_p1, B, l.N);
            at::mm_out(po, norms ? view(o_norm, B, DM) : x, l.w_in);
            proj.dense = base + o_p1;
        }
        fused = stream_w && L.bmx_decode_mixer_sums((int32_t)B, (int32_t)l.H, (int32_t)l.P) > 0;
        if (fused) {
            mix = bmx_mixer{};
            mix.batch = (int32_t)B, mix.nheads = (int32_t)l.H, mix.headdim = (int32_t)l.P, mix.ngroups = (int32_t)l.G, mix.norm_before_gate = l.before_gate;
            mix.nss = L.bmx_decode_mixer_sums((int32_t)B, (int32_t)l.H, (int32_t)l.P), mix.dt_min = l.dt_min, mix.dt_max = l.dt_max, mix.proj = proj, mix.planes = planes;
            mix.state = fptr(l.state), mix.window = fptr(l.window), mix.conv_w = fptr(&l.conv_w), mix.conv_b = fptr(&l.conv_b), mix.a = fptr(&l.a);
            mix.d = fptr(&l.d), mix.dt_bias = fptr(&l.dt_bias), mix.gamma = l.gamma.data_ptr(), mix.out = base + o_g;
            mix.ss = reinterpret_cast<float*>(base + o_ss);
            check(L.bmx_decode_mixer(&mix, st), "decode step (mixer)");
        } else {
            bm_conv_step_args ca;
            memset(&ca, 0, sizeof ca);
            ca.batch = (int32_t)B, ca.channels = (int32_t)l.V, ca.kernel = 4, ca.dtype = BM_DTYPE_BF16, ca.window = fptr(l.window), ca.weight = fptr(l.conv_w);
            ca.bias = fptr(l.conv_b), ca.out = base + o_x, ca.out_b = base + o_b, ca.out_c = base + o_c, ca.split_x = (int32_t)l.DI, ca.split_bc = (int32_t)(l.G * 128);
            check(L.bmx_decode_conv(&ca, &proj, (int32_t)l.DI, st), "decode step (conv)");
            bm_step2_args sa;
            memset(&sa, 0, sizeof sa);
            sa.batch = (int32_t)B, sa.nheads = (int32_t)l.H, sa.headdim = (int32_t)l.P, sa.state_rank = 128, sa.ngroups = (int32_t)l.G, sa.dtype = BM_DTYPE_BF16;
            sa.state = fptr(l.state), sa.x = base + o_x, sa.a = fptr(&l.a), sa.b = base + o_b, sa.c = base + o_c, sa.d = fptr(&l.d), sa.dt_bias = fptr(&l.dt_bias);
            sa.dt_min = l.dt_min, sa.dt_max = l.dt_max, sa.y = base + o_y;
            check(L.bmx_decode_state(&sa, &proj, (int32_t)(l.DI + l.V), st), "decode step (state)");
            bm_rmsnorm_gated_args na;
            memset(&na, 0, sizeof na);
            na.rows = (int32_t)B, na.width = (int32_t)l.DI, na.dtype = BM_DTYPE_BF16, na.norm_before_gate = l.before_gate, na.x_stride = (int32_t)l.DI, na.eps = eps;
            na.x = base + o_y, na.gamma = l.gamma.data_ptr(), na.out = base + o_g;
            check(L.bmx_decode_gated_norm(&na, &proj, planes, st), "decode step (gated norm)");
        }
        if (stream_w) {
            add = bmx_rows{};
            add.nslice = L.bmx_decode_slices((int32_t)B, (int32_t)l.DI, (int32_t)DM), add.slice = B * DM, add.ld = DM;
            float* p = reinterpret_cast<float*>(base + o_p2);
            check(L.bmx_decode_linear(base + o_g, planes, l.w_out.data_ptr(), p, (int32_t)B, (int32_t)l.DI, (int32_t)DM, add.nslice, status, 0, 0, st), "decode step (out-projection)");
            add.part = p;
            have_add = true;
        } else if (norms) {
            out.addmm_(view(o_g, B, l.DI), l.w_out);   // in place on the residual stream
        } else if (residual) {
            at::addmm_out(out, *residual, view(o_g, B, l.DI), l.w_out);
        } else {
            at::mm_out(out, view(o_g, B, l.DI), l.w_out);
        }
    }
    if (stream_w) check(L.bmx_decode_norm(xres, xres32, &add, fused ? &mix : nullptr, nullptr, eps, nullptr, out.data_ptr(), nullptr, 1, (int32_t)B, (int32_t)DM, 0, st), "decode step (residual)");
    if (check_status) {
        c10::cuda::getCurrentCUDAStream().synchronize();
        check(L.bmx_chain_take_status(status), "decode step");
    }
    scope.reset();
    return wrap(out);
    END
}

// ---- Mamba-3 block (mamba3.h) ------------------------------------------------------------------------------------------
struct M3Block {
    Tensor w_in, dt_bias, d, b_norm, c_norm, b_bias, c_bias, w_out, mimo_x, mimo_z, mimo_o;
    bmx_m3_block g;
    int64_t DM, DI, N, NA;
};
// Tuple (w_in, dt_bias, d, b_norm, c_norm, b_bias, c_bias, w_out, mimo_x | None, mimo_z | None, mimo_o | None, nheads, state_rank,
// ngroups, mimo_rank, rope_dim, range, dt_min, dt_max, a_floor, eps); false when the fused kernels do not cover the block.
bool read_m3(PyObject* tup, const Tensor& u, M3Block& b) {
    Tensor* ts[] = {&b.w_in, &b.dt_bias, &b.d, &b.b_norm, &b.c_norm, &b.b_bias, &b.c_bias, &b.w_out, &b.mimo_x, &b.mimo_z, &b.mimo_o};
    if (!PyTuple_Check(tup) || PyTuple_GET_SIZE(tup) != 21) return false;
    for (int i = 0; i < 11; ++i) {
        PyObject* o = PyTuple_GET_ITEM(tup, i);
        if (THPVariable_CheckExact(o)) *ts[i] = THPVariable_Unpack(o);
        else if (o != Py_None || i < 8) return false;
    }
    int64_t iv[5];
    double fv[5];
    for (int i = 0; i < 5; ++i) iv[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(tup, 11 + i));
    for (int i = 0; i < 5; ++i) fv[i] = PyFloat_AsDouble(PyTuple_GET_ITEM(tup, 16 + i));
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    const int64_t H = iv[0], R = iv[1], G = iv[2], M = iv[3], rope = iv[4];
    if (H < 1 || R < 1 || G < 1 || M < 1 || H % G || rope < 0 || rope > R || rope % 2 || b.w_out.dim() != 2) return false;
    b.DI = b.w_out.size(0), b.DM = b.w_out.size(1), b.NA = std::max<int64_t>(rope / 2, 1);
    const int64_t P = b.DI / H;
    b.N = 2 * b.DI + 2 * M * G * R + 3 * H + b.NA;
    if (P * H != b.DI || P % 4 || R % 4 || b.N % 4 || b.DI > 1 << 20) return false;
    const auto f = at::kFloat;
    const bool mimo = M > 1;
    if (!dense(b.w_in, f, {b.DM, b.N}, u) || !dense(b.w_out, f, {b.DI, b.DM}, u) || !dense(b.dt_bias, f, {H}, u) || !dense(b.d, f, {H}, u) ||
        !dense(b.b_norm, f, {R}, u) || !dense(b.c_norm, f, {R}, u) || !dense(b.b_bias, f, {H, M, R}, u) || !dense(b.c_bias, f, {H, M, R}, u) ||
        (b.mimo_x.defined() && !dense(b.mimo_x, f, {H, M, P}, u)) || (mimo && (!dense(b.mimo_z, f, {H, M, P}, u) || !dense(b.mimo_o, f, {H, M, P}, u))))
        return false;
    bmx_m3_block& g = b.g;
    memset(&g, 0, sizeof g);
    g.nheads = (int32_t)H, g.headdim = (int32_t)P, g.state_rank = (int32_t)R, g.ngroups = (int32_t)G, g.mimo_rank = (int32_t)M, g.rope_dim = (int32_t)rope;
    g.range = (float)fv[0], g.dt_min = (float)fv[1], g.dt_max = (float)fv[2], g.a_floor = (float)fv[3], g.eps = (float)fv[4];
    g.ld = b.N, g.dt_bias = fptr(&b.dt_bias), g.d = fptr(&b.d), g.b_norm = fptr(&b.b_norm), g.c_norm = fptr(&b.c_norm);
    g.b_bias = fptr(&b.b_bias), g.c_bias = fptr(&b.c_bias), g.mimo_x = b.mimo_x.defined() ? fptr(&b.mimo_x) : nullptr;
    g.mimo_z = mimo ? fptr(&b.mimo_z) : nullptr, g.mimo_o = mimo ? fptr(&b.mimo_o) : nullptr;
    return true;
}
bool m3_cache(const M3Block& b, const Tensor& u, const Tensor* ssm, const Tensor* k, const Tensor* v, const Tensor* angle) {
    const bmx_m3_block& g = b.g;
    const auto f = at::kFloat;
    const int64_t B = u.size(0);
    return ssm && k && v && angle && dense(*ssm, f, {B, g.nheads, g.headdim, g.state_rank}, u) && dense(*k, f, {B, g.mimo_rank, g.nheads, g.state_rank}, u) &&
           dense(*v, f, {B, g.nheads, g.headdim}, u) && dense(*angle, f, {B, g.nheads, b.NA}, u);
}

// block, u [b, s, d_model], ssm | None, k, v, angle, chunk_len -> (out, ssm, k, v, angle), or None when not covered.
// Mamba3::forward_single_ssd; ssm = None is the zero cache.
FN(m3_forward) {
    BEGIN
    PyObject* tup = A.next();
    const Tensor &u = *A.tensor("u"), *ssm = A.tensor("ssm", true), *k = A.tensor("k", true), *v0 = A.tensor("v", true), *angle = A.tensor("angle", true);
    const int64_t chunk = A.num();
    M3Block b;
    if (!A.exact || autocasting() || u.dim() != 3 || u.size(1) < 1 || !read_m3(tup, u, b) || b.g.state_rank % 16) return none();
    const int64_t B = u.size(0), S = u.size(1), H = b.g.nheads, P = b.g.headdim, R = b.g.state_rank, M = b.g.mimo_rank;
    if (B < 1 || !dense(u, at::kFloat, {B, S, b.DM}, u) || (ssm != nullptr && !m3_cache(b, u, ssm, k, v0, angle))) return none();
    if (elsewhere(u) || 2 * M * b.g.ngroups * R * 4 > 48 * 1024) return none();
    const auto f = at::kFloat;
    std::optional<NoGil> scope;   // until the results are wrapped
    scope.emplace();
    void* st = stream();
    Tensor proj = at::mm(u.view({B * S, b.DM}), b.w_in);
    b.g.batch = (int32_t)B, b.g.seqlen = (int32_t)S, b.g.proj = fptr(&proj);
    // per-step scalars and rot in one buffer
    const int64_t bsh = (B * S * H + 63) / 64 * 64;
    Tensor sc = empty({4 * bsh + B * S * b.NA}, f, u), v = empty({B, S, M, H, P}, f, u);
    float *dt = fptr(sc), *da = dt + bsh, *gamma = da + bsh, *scale = gamma + bsh, *rot = scale + bsh;
    check(L.bmx_m3_coefficients(&b.g, dt, da, gamma, scale, fptr(v), rot, st), "Mamba-3 block (coefficients)");
    Tensor last = empty({B, H, b.NA}, f, u), theta = empty({B, S, H, b.NA}, f, u);
    bm_angle_cumsum_args aa;
    memset(&aa, 0, sizeof aa);
    aa.batch = (int32_t)B, aa.seqlen = (int32_t)S, aa.nheads = (int32_t)H, aa.nangles = (int32_t)b.NA, aa.range = b.g.range, aa.rot = rot, aa.dt = dt;
    aa.prev = ssm ? fptr(angle) : nullptr, aa.theta = fptr(theta), aa.last = fptr(last);
    check(L.bm_angle_cumsum(&aa, st), "bm_angle_cumsum");
    Tensor bm = empty({B, S, M, H, R}, f, u), cm = empty({B, S, M, H, R}, f, u);
    bm_mamba3_bc_prep_args pa;
    memset(&pa, 0, sizeof pa);
    pa.batch = (int32_t)B, pa.seqlen = (int32_t)S, pa.mimo_rank = (int32_t)M, pa.ngroups = b.g.ngroups, pa.nheads = (int32_t)H, pa.state_rank = (int32_t)R;
    pa.dtype = BM_DTYPE_F32, pa.raw_stride = (int32_t)b.N, pa.rope_dim = b.g.rope_dim, pa.pairwise = M == 1, pa.eps = b.g.eps;
    pa.b_raw = fptr(proj) + 2 * b.DI, pa.c_raw = fptr(proj) + 2 * b.DI + M * b.g.ngroups * R, pa.b_gamma = b.g.b_norm, pa.c_gamma = b.g.c_norm;
    pa.b_bias = b.g.b_bias, pa.c_bias = b.g.c_bias, pa.angles = b.g.rope_dim > 0 ? fptr(&theta) : nullptr, pa.b_out = fptr(bm), pa.c_out = fptr(cm);
    check(L.bm_mamba3_bc_prep(&pa, st), "bm_mamba3_bc_prep");
    Tensor h0;
    if (ssm != nullptr) {
        h0 = empty({B, H, P, R}, f, u);
        check(L.bmx_m3_seed(&b.g, dt, gamma, fptr(ssm), fptr(k), fptr(v0), fptr(h0), st), "Mamba-3 block (initial state)");
    }
    Tensor y = empty({B, S, M, H, P}, f, u), hf = empty({B, H, P, R}, f, u);
    bm_ssd3_fwd_args fa;
    memset(&fa, 0, sizeof fa);
    fa.batch = (int32_t)B, fa.seqlen = (int32_t)S, fa.nheads = (int32_t)H, fa.headdim = (int32_t)P, fa.state_rank = (int32_t)R, fa.mimo_rank = (int32_t)M;
    fa.chunk_len = (int32_t)chunk, fa.dtype = BM_DTYPE_F32, fa.v = fptr(v), fa.da = da, fa.b = fptr(bm), fa.c = fptr(cm), fa.gamma = gamma, fa.scale = scale;
    fa.h0 = ssm ? fptr(&h0) : nullptr, fa.y = fptr(y), fa.h_final = fptr(hf);
    with_workspace(L.bm_ssd3_fwd_workspace_bytes(&fa), L.bmx_ssd3_fwd_least_bytes(&fa), u, "bm_ssd3_single_fwd", nullptr,
                   [&](void* ws, size_t n) { return L.bm_ssd3_single_fwd(&fa, ws, n, st); });
    Tensor g = empty({B * S, b.DI}, f, u), kl = empty({B, M, H, R}, f, u), vl = empty({B, H, P}, f, u);
    check(L.bmx_m3_tail(&b.g, fptr(&y), fptr(&bm), fptr(g), fptr(kl), fptr(vl), st), "Mamba-3 block (gate)");
    Tensor out = at::mm(g, b.w_out).view({B, S, b.DM});
    scope.reset();
    return tuple({wrap(out), wrap(hf), wrap(kl), wrap(vl), wrap(last)});
    END
}

// block, u [b, d_model], ssm, k, v, angle (updated in place) -> out [b, d_model], or None when not covered.
// Mamba3::step_double_ssd.
FN(m3_step) {
    BEGIN
    PyObject* tup = A.next();
    const Tensor &u = *A.tensor("u"), *ssm = A.tensor("ssm"), *k = A.tensor("k"), *v = A.tensor("v"), *angle = A.tensor("angle");
    M3Block b;
    if (!A.exact || autocasting() || u.dim() != 2 || !read_m3(tup, u, b)) return none();
    const int64_t B = u.size(0);
    b.g.batch = (int32_t)B, b.g.seqlen = 1;
    if (B < 1 || !dense(u, at::kFloat, {B, b.DM}, u) || !m3_cache(b, u, ssm, k, v, angle) || !L.bmx_m3_step_covers(&b.g) || elsewhere(u)) return none();
    Tensor out;
    {
        NoGil scope;
        Tensor proj = at::mm(u, b.w_in), g = empty({B, b.DI}, at::kFloat, u);
        b.g.proj = fptr(&proj);
        check(L.bmx_m3_step(&b.g, fptr(*ssm), fptr(*k), fptr(*v), fptr(*angle), fptr(g), stream()), "Mamba-3 step");
        out = at::mm(g, b.w_out);
    }
    return wrap(out);
    END
}

// ---- module ----------------------------------------------------------------------------------------------------------
// (no arguments) -> device status of the last SSD call on the current device and stream, or of the decode steps on the device;
// 0 when there was none
FN(workspace_status) {
    BEGIN
    (void)A;
    int32_t status = BM_OK;
    {
        NoGil scope;
        const int device = (int)c10::cuda::current_device();
        c10::cuda::getCurrentCUDAStream().synchronize();
        status = L.bmx_chain_take_status(chain_status(device));
        if (Workspace* w = status == BM_OK ? find_workspace(device, false) : nullptr) {
            std::lock_guard<std::mutex> lock(w->m);
            if (w->t.defined()) status = L.bm_workspace_status(w->t.data_ptr(), stream());
        }
    }
    return PyLong_FromLong(status);
    END
}

// path of libbm_b200, BmError class
FN(init) {
    BEGIN
    const char* path = PyUnicode_AsUTF8(A.next());
    if (path == nullptr) return nullptr;
    void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (h == nullptr) {
        PyErr_Format(PyExc_ImportError, "%s: %s", path, dlerror());
        return nullptr;
    }
#define X(n)                                                                       \
    L.n = reinterpret_cast<decltype(L.n)>(dlsym(h, #n));                           \
    if (L.n == nullptr) {                                                          \
        PyErr_Format(PyExc_ImportError, "%s: symbol %s is missing", path, #n);     \
        return nullptr;                                                            \
    }
    BM_ENTRY_POINTS(X)
#undef X
    PyObject* err = A.next();
    Py_INCREF(err);
    Py_XSETREF(g_bm_error, err);
    Py_RETURN_NONE;
    END
}

PyMethodDef kMethods[] = {
#define M(n) {#n, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(n)), METH_FASTCALL, nullptr}
    M(init), M(ssd2_fwd), M(ssd2_bwd), M(step2), M(conv_step), M(conv1d_silu_fwd), M(rmsnorm_gated), M(selscan1_fwd), M(step1),
    M(mamba3_bc_prep), M(ssd3_fwd), M(ssd3_bwd), M(angle_cumsum), M(step3), M(workspace_status), M(m2_decode), M(m3_forward), M(m3_step),
#undef M
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Host path of the burn_mamba_b200 calls.", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
