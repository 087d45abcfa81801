// Host path of the operators: argument checks, buffers, plan lookup and launches in native code.
//
// A call of an operator costs a few microseconds of GPU time at serving sizes, so what the host does per call decides the
// rate: the same checks and launches in Python (tensor attributes, a device context manager, ctypes with twenty arguments)
// took 25 - 45 us per operator and 1.75 ms for the 72 launches of a 12-layer encoder on 128 tokens.  This module takes the
// Python arguments once, works on at::Tensor, and calls the C ABI (include/stof_b200.h) through function pointers of the
// library that the ctypes layer loaded; the encoder and decoder stacks walk their layers here without returning to Python.
//
// Python keeps what is decided once per mask: the attention plan and its schedule (attention.plan_for_call).  A decided plan
// is remembered here under the identity of its index tensors, so that later calls find it without Python.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <sched.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <optional>
#include <string>
#include <vector>

#include "../../../include/stof_b200.h"

namespace {

// ------------------------------------------------------------------------------------------ errors
struct StofFail { std::string text; };
struct PythonFail {};                        // a Python exception is already set

[[noreturn]] void fail(const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    throw StofFail{buf};
}

PyObject* g_error = nullptr;                 // StofError
PyObject* g_status_word = nullptr;           // device index -> int32 tensor
PyObject* g_check_status = nullptr;          // (device index, what): reads the word, clears it and raises
PyObject* g_plan_for_call = nullptr;         // (index tensors, seq, batch, heads, block_m, block_n) -> (plan, schedule, blocks, final)

template <class F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const StofFail& e) {
        PyErr_SetString(g_error != nullptr ? g_error : PyExc_RuntimeError, e.text.c_str());
    } catch (const PythonFail&) {
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// ------------------------------------------------------------------------------------------ the library
struct Api {
    decltype(&stof_last_error) last_error;
    decltype(&stof_mask_workspace_bytes) mask_workspace_bytes;
    decltype(&stof_mask_classify_notify) mask_classify_notify;
    decltype(&stof_mask_fill) mask_fill;
    decltype(&stof_block_attn) block_attn;
    decltype(&stof_block_attn_scheduled) block_attn_scheduled;
    decltype(&stof_gemm_bias_act) gemm_bias_act;
    decltype(&stof_gemm_bias_residual_layernorm) gemm_ln;
    decltype(&stof_bias_residual_layernorm) layernorm;
} api = {};

void check(int rc, const char* what) {
    if (rc != 0) fail("%s failed (code %d): %s", what, rc, api.last_error());
}

// The GIL is free while the library launches and torch copies or allocates: where the queue of launches is full they wait for the GPU,
// and what the GPU waits for may need Python (a host callback in the stream, another thread).  One that stands inside another does
// nothing; whoever needs several calls in a row takes it once around them, as every turn with the lock may have to wait for a thread
// that computes in Python.
struct Released {
    PyThreadState* ts = PyGILState_Check() ? PyEval_SaveThread() : nullptr;
    Released() = default;
    Released(const Released&) = delete;
    ~Released() { if (ts != nullptr) PyEval_RestoreThread(ts); }
};
template <class F>
auto released(F&& f) {
    const Released gil;
    return f();
}
template <class F, class... A>
void call(const char* what, F* f, A... args) {
    int rc;
    {
        const Released gil;
        rc = f(args...);
    }
    check(rc, what);                         // the error text is the calling thread's own
}
at::Tensor packed(const at::Tensor& t) {
    if (t.is_contiguous()) return t;
    const Released gil;
    return t.contiguous();
}

// ------------------------------------------------------------------------------------------ arguments
// A tensor argument (nullptr for None); anything else is a TypeError.
const at::Tensor* tensor_arg(PyObject* o, const char* what) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s: a tensor expected, got %s", what, Py_TYPE(o)->tp_name);
        throw PythonFail{};
    }
    return &THPVariable_Unpack(o);
}
const at::Tensor& tensor_needed(PyObject* o, const char* what) {
    const at::Tensor* t = tensor_arg(o, what);
    if (t == nullptr) {
        PyErr_Format(PyExc_TypeError, "%s: a tensor expected, got None", what);
        throw PythonFail{};
    }
    return *t;
}
// a whole number as int(o) gives it, for what is not an int itself (a size that was computed as a float)
long long_arg(PyObject* o) {
    PyObject* whole = PyLong_Check(o) ? o : PyNumber_Long(o);
    if (whole == nullptr) throw PythonFail{};
    const long v = PyLong_AsLong(whole);
    if (whole != o) Py_DECREF(whole);
    if (v == -1 && PyErr_Occurred()) throw PythonFail{};
    return v;
}
double double_arg(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PythonFail{};
    return v;
}
void need_args(Py_ssize_t got, Py_ssize_t want, const char* what) {
    if (got != want) {
        PyErr_Format(PyExc_TypeError, "%s: %zd arguments expected, got %zd", what, want, got);
        throw PythonFail{};
    }
}
PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
PyObject* same(PyObject* o) {
    Py_INCREF(o);
    return o;
}

inline bool is_half(const at::Tensor& t) { return t.scalar_type() == at::kHalf; }
void need_cuda(const at::Tensor* t) {
    if (t != nullptr && !t->is_cuda()) fail("stof_b200 operators need CUDA tensors (there is no CPU fallback)");
}

// ------------------------------------------------------------------------------------------ device, stream, status word
constexpr int MAX_DEVICES = 64;
int* g_status_ptr[MAX_DEVICES] = {};         // the words are tensors that the Python layer keeps for good

int* status_ptr(int dev) {
    if (dev < 0 || dev >= MAX_DEVICES) fail("device ordinal %d out of range", dev);
    if (g_status_ptr[dev] == nullptr) {
        PyObject* w = PyObject_CallFunction(g_status_word, "i", dev);
        if (w == nullptr) throw PythonFail{};
        g_status_ptr[dev] = static_cast<int*>(tensor_needed(w, "status word").data_ptr());
        Py_DECREF(w);
    }
    return g_status_ptr[dev];
}

struct Launch {                              // device made current, its current stream, its status word
    c10::cuda::CUDAGuard guard;
    void* stream;
    int* status;
    explicit Launch(const at::Tensor& t)
        : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.get_device()).stream()), status(status_ptr(t.get_device())) {}
};

// A new tensor on t's device, without the dispatcher's round
at::Tensor make(at::IntArrayRef shape, at::ScalarType type, const at::Tensor& t) {
    const Released gil;
    return at::detail::empty_cuda(shape, type, t.device(), std::nullopt);
}

// ------------------------------------------------------------------------------------------ matrices
struct Rows {                                // a (..., C) tensor seen as rows of C with a contiguous last dimension
    at::Tensor keep;                         // the copy, where one had to be made
    const void* ptr;
    int64_t rows, cols, ld;
};
Rows as_rows(const at::Tensor& t) {
    Rows r;
    const int64_t d = t.dim();
    if (d == 0) fail("a tensor with at least one dimension expected");
    r.cols = t.size(d - 1);
    if (t.is_contiguous()) {
        r.rows = r.cols > 0 ? t.numel() / r.cols : 0;
        r.ld = d == 1 ? r.cols : (d == 2 ? t.stride(0) : r.cols);
        if (r.rows <= 1 && r.ld < r.cols) r.ld = r.cols;
        r.ptr = t.data_ptr();
        return r;
    }
    {
        const Released gil;
        r.keep = (t.stride(d - 1) != 1 ? t.contiguous() : t).reshape({-1, r.cols});
    }
    r.rows = r.keep.size(0);
    r.ld = r.keep.stride(0);
    r.ptr = r.keep.data_ptr();
    return r;
}

// A (N) vector operand of a fused operator: fp16, any shape with N elements.  A copy, where one is needed, goes into `keep`.
const void* vector_arg(const at::Tensor* v, int64_t n, at::Tensor& keep, const char* text) {
    if (v == nullptr) return nullptr;
    if (v->numel() != n || !is_half(*v)) fail("%s", text);
    if (v->is_contiguous()) return v->data_ptr();
    keep = packed(*v).reshape({-1});
    return keep.data_ptr();
}

// The output: made here, or the caller's, which has to be viewable as contiguous rows
struct Out {
    at::Tensor made;
    void* ptr;
    int64_t ld;
};
Out output_rows(const at::Tensor* out, const at::Tensor& like, int64_t rows, int64_t cols, const char* op) {
    Out o;
    if (out == nullptr) {
        c10::SmallVector<int64_t, 5> shape(like.sizes().begin(), like.sizes().end());
        shape.back() = cols;
        o.made = make(shape, at::kHalf, like);
        o.ptr = o.made.data_ptr();
        o.ld = cols;
        return o;
    }
    if (!is_half(*out) || out->numel() != rows * cols || out->dim() == 0 || out->size(-1) != cols)
        fail("%s: out must be float16 with %lld rows of %lld", op, static_cast<long long>(rows), static_cast<long long>(cols));
    const Rows r = as_rows(*out);
    if (r.ptr != out->data_ptr() || (cols > 1 && out->stride(-1) != 1)) fail("%s: output must be viewable as contiguous rows", op);
    o.ptr = const_cast<void*>(r.ptr);
    o.ld = r.ld;
    return o;
}

struct Weight {
    at::Tensor keep;
    const void* ptr;
    int64_t k, n, ld;
};
Weight weight_arg(const at::Tensor& w) {
    Weight r;
    r.k = w.size(0);
    r.n = w.size(1);
    if (w.stride(1) == 1) {
        r.ptr = w.data_ptr();
        r.ld = w.stride(0);
    } else {
        r.keep = packed(w);
        r.ptr = r.keep.data_ptr();
        r.ld = r.keep.stride(0);
    }
    return r;
}

// a (..., K) @ w (K, N) + bias, with an epilogue; the result goes into `out` or a new tensor, which is returned
at::Tensor gemm_core(const Launch& l, const at::Tensor& a, const at::Tensor& w, const at::Tensor* bias, int epilogue, const at::Tensor* residual,
                     const at::Tensor* out) {
    if (!is_half(a) || !is_half(w)) fail("gemm: float16 operands expected");
    if (w.dim() != 2) fail("gemm: weight must be (K, N)");
    const Rows x = as_rows(a);
    const Weight m = weight_arg(w);
    if (x.cols != m.k) fail("gemm: inner dimensions differ (%lld vs %lld)", static_cast<long long>(x.cols), static_cast<long long>(m.k));
    at::Tensor kept_bias;
    const void* b = vector_arg(bias, m.n, kept_bias, "gemm: bias must be a float16 vector of length N");
    const Out c = output_rows(out, a, x.rows, m.n, "gemm");
    Rows r{{}, nullptr, 0, 0, 0};
    if (residual != nullptr) {
        if (!is_half(*residual)) fail("gemm: residual must be float16 of the output's shape");
        r = as_rows(*residual);
        if (r.rows != x.rows || r.cols != m.n) fail("gemm: residual must be float16 of the output's shape");
    }
    call("stof_gemm_bias_act", api.gemm_bias_act, x.ptr, x.ld, m.ptr, m.ld, b, r.ptr, r.ld, c.ptr, c.ld, static_cast<int>(x.rows), static_cast<int>(m.n),
         static_cast<int>(m.k), epilogue, l.status, l.stream);
    return c.made;
}

at::Tensor gemm_ln_core(const Launch& l, const at::Tensor& a, const at::Tensor& w, const at::Tensor* bias, const at::Tensor* residual,
                        const at::Tensor* gamma, const at::Tensor* beta, double eps, const at::Tensor* out) {
    if (!is_half(a) || !is_half(w) || w.dim() != 2) fail("gemm+layernorm: float16 operands and a (K, N) weight expected");
    const Rows x = as_rows(a);
    const Weight m = weight_arg(w);
    if (x.cols != m.k) fail("gemm+layernorm: inner dimensions differ (%lld vs %lld)", static_cast<long long>(x.cols), static_cast<long long>(m.k));
    static const char* text = "gemm+layernorm: bias/gamma/beta must be float16 vectors of length N";
    at::Tensor kept[3];
    const void* b = vector_arg(bias, m.n, kept[0], text);
    const void* g = vector_arg(gamma, m.n, kept[1], text);
    const void* t = vector_arg(beta, m.n, kept[2], text);
    const Out c = output_rows(out, a, x.rows, m.n, "gemm+layernorm");
    Rows r{{}, nullptr, 0, 0, 0};
    if (residual != nullptr) {
        if (!is_half(*residual)) fail("gemm+layernorm: residual must be float16 of the output's shape");
        r = as_rows(*residual);
        if (r.rows != x.rows || r.cols != m.n) fail("gemm+layernorm: residual must be float16 of the output's shape");
    }
    call("stof_gemm_bias_residual_layernorm", api.gemm_ln, x.ptr, x.ld, m.ptr, m.ld, b, r.ptr, r.ld, g, t, static_cast<float>(eps), c.ptr, c.ld,
         static_cast<int>(x.rows), static_cast<int>(m.n), static_cast<int>(m.k), l.status, l.stream);
    return c.made;
}

at::Tensor layernorm_core(const Launch& l, const at::Tensor& a, const at::Tensor* bias, const at::Tensor* residual, const at::Tensor* gamma,
                          const at::Tensor* beta, double eps, const at::Tensor* out) {
    if (!is_half(a)) fail("layernorm: float16 input expected");
    const Rows x = as_rows(a);
    Rows r{{}, nullptr, 0, 0, 0};
    if (residual != nullptr) {
        if (!is_half(*residual)) fail("layernorm: residual must be float16 of the input's shape");
        r = as_rows(*residual);
        if (r.rows != x.rows || r.cols != x.cols) fail("layernorm: residual must be float16 of the input's shape");
    }
    static const char* text = "layernorm: bias/gamma/beta must be float16 vectors of length hidden";
    at::Tensor kept[3];
    const void* b = vector_arg(bias, x.cols, kept[0], text);
    const void* g = vector_arg(gamma, x.cols, kept[1], text);
    const void* t = vector_arg(beta, x.cols, kept[2], text);
    const Out y = output_rows(out, a, x.rows, x.cols, "layernorm");
    call("stof_bias_residual_layernorm", api.layernorm, x.ptr, x.ld, b, r.ptr, r.ld, g, t, static_cast<float>(eps), y.ptr, y.ld, static_cast<int>(x.rows),
         static_cast<int>(x.cols), l.status, l.stream);
    return y.made;
}

// ------------------------------------------------------------------------------------------ attention plans
// A decided plan under the identity of its index: storage, version counter and length of the four index tensors (which the
// entry keeps alive, so that no other tensor can take their addresses), shape and block sizes.  Rewrites that torch does not
// see are announced through forget().  A few dozen entries, the one used last in front.
struct PlanKey {
    const void* ptr[4];
    int64_t version[4], numel[4];
    int64_t seq, batch, heads, bm, bn, dev;
    bool operator==(const PlanKey& o) const {
        for (int i = 0; i < 4; ++i)
            if (ptr[i] != o.ptr[i] || version[i] != o.version[i] || numel[i] != o.numel[i]) return false;
        return seq == o.seq && batch == o.batch && heads == o.heads && bm == o.bm && bn == o.bn && dev == o.dev;
    }
};
struct PlanEntry {
    PlanKey key;
    at::Tensor index[4], plan, schedule;     // schedule: undefined when the default deal is used
    int blocks;
    bool decided;                            // remembered: a later lookup gives the same
};
constexpr size_t MAX_PLANS = 32;
std::vector<PlanEntry>& plans() {
    static std::vector<PlanEntry>* v = new std::vector<PlanEntry>();     // never destroyed: tensors must not outlive the runtime
    return *v;
}

struct Index {
    const at::Tensor* t[4];                  // full_row_ptr, full_col_idx, part_row_ptr, part_col_idx
    PyObject* o[4];
    const at::Tensor* tiles;                 // part_block_mask
};

PlanEntry plan_lookup(const Index& ix, int64_t seq, int64_t batch, int64_t heads, int64_t bm, int64_t bn, int64_t dev) {
    if (bm <= 0 || bn <= 0) fail("block attention: block sizes must be positive");
    // On every call, known index or not: base[:n] and base[::2] of one tensor agree in all that the key holds
    for (int i = 0; i < 4; ++i)
        if (ix.t[i]->scalar_type() != at::kInt || !ix.t[i]->is_contiguous()) fail("block attention: index tensors must be contiguous int32");
    if (ix.t[0]->numel() != seq / bm + 1 || ix.t[2]->numel() != seq / bm + 1)
        fail("block attention: row pointer arrays must have S / BLOCK_M + 1 entries");
    PlanKey key;
    bool keyed = true;
    for (int i = 0; i < 4; ++i) {
        key.ptr[i] = ix.t[i]->data_ptr();
        key.numel[i] = ix.t[i]->numel();
        keyed = keyed && !ix.t[i]->is_inference();
        key.version[i] = keyed ? static_cast<int64_t>(ix.t[i]->_version()) : 0;
    }
    key.seq = seq; key.batch = batch; key.heads = heads; key.bm = bm; key.bn = bn; key.dev = dev;
    auto& all = plans();
    if (keyed)
        for (size_t i = 0; i < all.size(); ++i)
            if (all[i].key == key) {
                if (i > 0) std::rotate(all.begin(), all.begin() + static_cast<long>(i), all.begin() + static_cast<long>(i) + 1);
                return all[0];
            }
    PyObject* r = PyObject_CallFunction(g_plan_for_call, "OOOOLLLLL", ix.o[0], ix.o[1], ix.o[2], ix.o[3], static_cast<long long>(seq),
                                        static_cast<long long>(batch), static_cast<long long>(heads), static_cast<long long>(bm),
                                        static_cast<long long>(bn));
    if (r == nullptr) throw PythonFail{};
    PyObject *plan, *schedule;
    int blocks, final_;
    if (!PyArg_ParseTuple(r, "OOip", &plan, &schedule, &blocks, &final_)) {
        Py_DECREF(r);
        throw PythonFail{};
    }
    PlanEntry e;
    e.key = key;
    for (int i = 0; i < 4; ++i) e.index[i] = *ix.t[i];
    e.plan = tensor_needed(plan, "plan");
    if (schedule != Py_None) e.schedule = tensor_needed(schedule, "schedule");
    e.blocks = blocks;
    e.decided = keyed && final_;
    Py_DECREF(r);
    if (e.decided) {
        if (all.size() >= MAX_PLANS) all.pop_back();
        all.insert(all.begin(), e);
    }
    return e;
}

struct HeadView {                            // a (B, H, S, 64) view
    void* ptr;
    long long stride[3];
};

void attention_launch(const Launch& l, const PlanEntry& e, const HeadView& q, const HeadView& k, const HeadView& v, const HeadView& out,
                      const at::Tensor* tiles, int head_dim, float scale) {
    const int B = static_cast<int>(e.key.batch), H = static_cast<int>(e.key.heads), S = static_cast<int>(e.key.seq);
    const int bm = static_cast<int>(e.key.bm), bn = static_cast<int>(e.key.bn);
    const int* prp = static_cast<const int*>(e.index[2].data_ptr());
    const void* pbm = tiles != nullptr ? tiles->data_ptr() : nullptr;
    if (e.schedule.defined())
        call("stof_block_attn", api.block_attn_scheduled, q.ptr, k.ptr, v.ptr, out.ptr, B, H, S, head_dim, q.stride, k.stride, v.stride, out.stride,
             prp, pbm, e.plan.data_ptr(), bm, bn, 4, scale, static_cast<const int*>(e.schedule.data_ptr()), e.blocks, l.status, l.stream);
    else
        call("stof_block_attn", api.block_attn, q.ptr, k.ptr, v.ptr, out.ptr, B, H, S, head_dim, q.stride, k.stride, v.stride, out.stride, prp, pbm,
             e.plan.data_ptr(), bm, bn, 4, scale, l.status, l.stream);
}

Index index_args(PyObject* const* a, const at::Tensor* tiles = nullptr) {
    Index ix;
    for (int i = 0; i < 4; ++i) {
        ix.o[i] = a[i];
        ix.t[i] = &tensor_needed(a[i], "block index");
    }
    ix.tiles = tiles != nullptr ? tiles : tensor_arg(a[4], "part_block_mask");
    need_cuda(ix.t[0]);
    need_cuda(ix.t[2]);
    if (ix.tiles != nullptr && (!is_half(*ix.tiles) || !ix.tiles->is_contiguous()))
        fail("block attention: part_block_mask must be contiguous float16");
    return ix;
}

HeadView head_view(const at::Tensor& t) {
    return HeadView{t.data_ptr(), {t.stride(0), t.stride(1), t.stride(2)}};
}

void attention_core(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& out, const Index& ix, int64_t bm, int64_t bn,
                    std::optional<double> softmax_scale = std::nullopt) {
    const at::Tensor* all[4] = {&q, &k, &v, &out};
    for (const at::Tensor* t : all) need_cuda(t);
    for (const at::Tensor* t : all)
        if (!is_half(*t)) fail("block attention expects float16 q/k/v/out");
    if (q.dim() != 4) fail("block attention: q must be (B,H,S,D)");
    for (const at::Tensor* t : all) {
        if (t->sizes() != q.sizes()) fail("block attention: q, k, v and out must share one (B,H,S,D) shape");
        if (t->stride(3) != 1) fail("block attention: the head dimension must be contiguous");
    }
    const double scale = softmax_scale ? *softmax_scale : 1.0 / std::sqrt(static_cast<double>(q.size(3)));          // src/ops/src/block_attn_mask.cpp:32
    const Launch l(q);
    const PlanEntry e = plan_lookup(ix, q.size(2), q.size(0), q.size(1), bm, bn, q.get_device());
    attention_launch(l, e, head_view(q), head_view(k), head_view(v), head_view(out), ix.tiles, static_cast<int>(q.size(3)),
                     static_cast<float>(scale));
}

// ------------------------------------------------------------------------------------------ Python entry points
// gemm(a, w, bias, epilogue, residual, out) -> out
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 6, "gemm");
        const at::Tensor &x = tensor_needed(a[0], "gemm"), &w = tensor_needed(a[1], "gemm");
        const at::Tensor *bias = tensor_arg(a[2], "gemm"), *res = tensor_arg(a[4], "gemm"), *out = tensor_arg(a[5], "gemm");
        for (const at::Tensor* t : {&x, &w, bias, res, out}) need_cuda(t);
        const int epilogue = static_cast<int>(long_arg(a[3]));
        const Launch l(x);
        const at::Tensor made = released([&] { return gemm_core(l, x, w, bias, epilogue, res, out); });
        return out != nullptr ? same(a[5]) : wrap(made);
    });
}

// gemm_ln(a, w, bias, residual, gamma, beta, eps, out) -> out
PyObject* py_gemm_ln(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 8, "gemm_ln");
        const at::Tensor &x = tensor_needed(a[0], "gemm_ln"), &w = tensor_needed(a[1], "gemm_ln");
        const at::Tensor *v[4], *out = tensor_arg(a[7], "gemm_ln");
        for (int i = 0; i < 4; ++i) v[i] = tensor_arg(a[2 + i], "gemm_ln");
        for (const at::Tensor* t : {&x, &w, v[0], v[1], v[2], v[3], out}) need_cuda(t);
        const double eps = double_arg(a[6]);
        const Launch l(x);
        const at::Tensor made = released([&] { return gemm_ln_core(l, x, w, v[0], v[1], v[2], v[3], eps, out); });
        return out != nullptr ? same(a[7]) : wrap(made);
    });
}

// layernorm(x, bias, residual, gamma, beta, eps, out) -> out
PyObject* py_layernorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 7, "layernorm");
        const at::Tensor& x = tensor_needed(a[0], "layernorm");
        const at::Tensor *v[4], *out = tensor_arg(a[6], "layernorm");
        for (int i = 0; i < 4; ++i) v[i] = tensor_arg(a[1 + i], "layernorm");
        for (const at::Tensor* t : {&x, v[0], v[1], v[2], v[3], out}) need_cuda(t);
        const double eps = double_arg(a[5]);
        const Launch l(x);
        const at::Tensor made = released([&] { return layernorm_core(l, x, v[0], v[1], v[2], v[3], eps, out); });
        return out != nullptr ? same(a[6]) : wrap(made);
    });
}

// attention(q, k, v, out, full_row_ptr, full_col_idx, part_row_ptr, part_col_idx, part_block_mask, block_m, block_n, scale) -> out;
// None as scale stands for 1 / sqrt(head_dim)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 12, "attention");
        attention_core(tensor_needed(a[0], "attention"), tensor_needed(a[1], "attention"), tensor_needed(a[2], "attention"),
                       tensor_needed(a[3], "attention"), index_args(a + 4), long_arg(a[9]), long_arg(a[10]),
                       a[11] != Py_None ? std::optional<double>(double_arg(a[11])) : std::nullopt);
        return same(a[3]);
    });
}

// attention_inplace(q, k, v, five index tensors, block_m, block_n) -> q, overwritten
PyObject* py_attention_inplace(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 10, "attention_inplace");
        const at::Tensor &q = tensor_needed(a[0], "attention"), &k = tensor_needed(a[1], "attention"), &v = tensor_needed(a[2], "attention");
        if (!q.is_contiguous()) fail("block_attn_mask: q must be contiguous (it is overwritten in place)");
        const at::Tensor kc = packed(k), vc = packed(v), tiles = packed(tensor_needed(a[7], "block index"));
        attention_core(q, kc, vc, q, index_args(a + 3, &tiles), long_arg(a[8]), long_arg(a[9]));
        return same(a[0]);
    });
}

// merged_attention(q, k, v, result or None, five index tensors, block_m, block_n) -> (B, S, H * D) result
PyObject* py_merged_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 11, "merged_attention");
        const at::Tensor &q = tensor_needed(a[0], "attention"), &k = tensor_needed(a[1], "attention"), &v = tensor_needed(a[2], "attention");
        const at::Tensor* result = tensor_arg(a[3], "attention");
        for (const at::Tensor* t : {&q, &k, &v, result}) need_cuda(t);
        if (q.dim() != 4) fail("row-wise attention: q must be (B,H,S,D)");
        const int64_t B = q.size(0), H = q.size(1), S = q.size(2), D = q.size(3);
        at::Tensor made;
        if (result == nullptr) {
            made = make({B, S, H * D}, q.scalar_type(), q);
        } else if (result->sizes() != at::IntArrayRef({B, S, H * D}) || !result->is_contiguous()) {
            fail("row-wise attention: result must be a contiguous (batch, S, heads*64) tensor");
        }
        const at::Tensor& r = result != nullptr ? *result : made;
        attention_core(q, k, v, r.as_strided({B, H, S, D}, {S * H * D, D, H * D, 1}), index_args(a + 4), long_arg(a[9]), long_arg(a[10]));
        return result != nullptr ? same(a[3]) : wrap(made);
    });
}

// forget(data_ptr): the index tensor at this address was rewritten behind torch's back
PyObject* py_forget(PyObject*, PyObject* arg) {
    const void* p = PyLong_AsVoidPtr(arg);
    if (p == nullptr && PyErr_Occurred()) return nullptr;
    auto& all = plans();
    for (size_t i = all.size(); i-- > 0;)
        for (int j = 0; j < 4; ++j)
            if (all[i].key.ptr[j] == p) {
                all.erase(all.begin() + static_cast<long>(i));
                break;
            }
    Py_RETURN_NONE;
}

// ------------------------------------------------------------------------------------------ encoder and decoder stacks
// A layer's weights, by attribute name, as tensors (the objects stay alive in the layer).  Biases, gamma and beta may be None: an
// undefined tensor, which `given` turns into the operators' nullptr.
struct LayerReader {
    PyObject* layer;
    at::Tensor vector(PyObject* name) const {
        PyObject* o = PyObject_GetAttr(layer, name);
        if (o == nullptr) throw PythonFail{};
        struct Drop { PyObject* o; ~Drop() { Py_DECREF(o); } } drop{o};
        const at::Tensor* t = tensor_arg(o, "layer weight");
        need_cuda(t);
        return t != nullptr ? *t : at::Tensor();
    }
    at::Tensor operator()(PyObject* name) const {
        const at::Tensor t = vector(name);
        if (!t.defined()) {
            PyErr_Format(PyExc_TypeError, "layer weight %U: a tensor expected, got None", name);
            throw PythonFail{};
        }
        return t;
    }
};
inline const at::Tensor* given(const at::Tensor& t) { return t.defined() ? &t : nullptr; }
#define STOF_NAME(s) ([] { static PyObject* n = PyUnicode_InternFromString(s); return n; }())

struct Stack {
    at::Tensor qkv, ctx, inter;
    at::Tensor y[4];
    PyObject* y_obj[4];
    int n_y;
    Index ix;
    int64_t heads, bm, bn;
    double eps;
};

void attention_sublayer(const Launch& l, const Stack& s, const PlanEntry& plan, const at::Tensor& x, const at::Tensor& wqkv, const at::Tensor& bqkv) {
    gemm_core(l, x, wqkv, given(bqkv), STOF_EPI_BIAS, nullptr, &s.qkv);
    const long long S = s.ctx.size(1), hid = s.ctx.size(2), D = hid / s.heads;
    char* base = static_cast<char*>(s.qkv.data_ptr());
    const HeadView q{base, {S * 3 * hid, D, 3 * hid}};
    const HeadView k{base + 2 * hid, {S * 3 * hid, D, 3 * hid}};
    const HeadView v{base + 4 * hid, {S * 3 * hid, D, 3 * hid}};
    const HeadView o{s.ctx.data_ptr(), {S * hid, D, hid}};
    attention_launch(l, plan, q, k, v, o, s.ix.tiles, static_cast<int>(D), static_cast<float>(1.0 / std::sqrt(static_cast<double>(D))));
}

void residual_layernorm(const Launch& l, bool fuse, const at::Tensor& a, const at::Tensor& w, const at::Tensor& bias, const at::Tensor& residual,
                        const at::Tensor& g, const at::Tensor& b, double eps, const at::Tensor& out) {
    if (fuse) {
        gemm_ln_core(l, a, w, given(bias), &residual, given(g), given(b), eps, &out);
    } else {
        gemm_core(l, a, w, given(bias), STOF_EPI_BIAS_RESIDUAL, &residual, &out);
        layernorm_core(l, out, nullptr, nullptr, given(g), given(b), eps, &out);
    }
}

// stack(layers, hidden, qkv, ctx, inter, (y buffers), five index tensors, block_m, block_n, heads, eps, activation epilogue,
//       fuse_layernorm, decoder) -> the buffer that holds the last layer's output
PyObject* py_stack(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 18, "stack");
        const at::Tensor& hidden = tensor_needed(a[1], "hidden");
        need_cuda(&hidden);
        if (hidden.dim() != 3) fail("encoder: hidden must be (B, S, hidden)");
        Stack s;
        s.qkv = tensor_needed(a[2], "qkv");
        s.ctx = tensor_needed(a[3], "ctx");
        s.inter = tensor_needed(a[4], "inter");
        s.n_y = static_cast<int>(PyTuple_GET_SIZE(a[5]));
        if (s.n_y < 1 || s.n_y > 4) fail("encoder: one to four hidden-state buffers expected, got %d", s.n_y);
        for (int i = 0; i < s.n_y; ++i) {
            s.y_obj[i] = PyTuple_GET_ITEM(a[5], i);
            s.y[i] = tensor_needed(s.y_obj[i], "y");
        }
        s.ix = index_args(a + 6);
        s.bm = long_arg(a[11]);
        s.bn = long_arg(a[12]);
        s.heads = long_arg(a[13]);
        s.eps = double_arg(a[14]);
        // the heads' views of qkv and ctx are made from D = hidden / heads below
        const int64_t hid = hidden.size(2);
        if (s.heads <= 0 || hid % s.heads != 0)
            fail("encoder: hidden size %lld is not a multiple of the %lld heads", static_cast<long long>(hid), static_cast<long long>(s.heads));
        const int act = static_cast<int>(long_arg(a[15]));
        const bool fuse = PyObject_IsTrue(a[16]) == 1, decoder = PyObject_IsTrue(a[17]) == 1;
        struct Attention { at::Tensor Wqkv, bqkv, Wo, bo, g, b; };
        struct Layer { Attention a[2]; at::Tensor W1, bi1, W2, bi2, g2, b2; };
        const Py_ssize_t count = PySequence_Size(a[0]);
        if (count < 0) throw PythonFail{};
        std::vector<Layer> layers(static_cast<size_t>(count));
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject* layer = PySequence_GetItem(a[0], i);
            if (layer == nullptr) throw PythonFail{};
            struct Drop { PyObject* o; ~Drop() { Py_DECREF(o); } } drop{layer};
            const LayerReader w{layer};
            Layer& m = layers[static_cast<size_t>(i)];
            if (decoder) {
                m.a[0] = {w(STOF_NAME("Wqkv_a")), w.vector(STOF_NAME("bqkv_a")), w(STOF_NAME("Wo_a")), w.vector(STOF_NAME("bo_a")), w.vector(STOF_NAME("g_a")),
                          w.vector(STOF_NAME("b_a"))};
                m.a[1] = {w(STOF_NAME("Wqkv_c")), w.vector(STOF_NAME("bqkv_c")), w(STOF_NAME("Wo_c")), w.vector(STOF_NAME("bo_c")), w.vector(STOF_NAME("g_c")),
                          w.vector(STOF_NAME("b_c"))};
            } else {
                m.a[0] = {w(STOF_NAME("Wqkv")), w.vector(STOF_NAME("bqkv")), w(STOF_NAME("Wo")), w.vector(STOF_NAME("bo")), w.vector(STOF_NAME("g1")),
                          w.vector(STOF_NAME("b1"))};
            }
            m.W1 = w(STOF_NAME("W1"));
            m.bi1 = w.vector(STOF_NAME("bi1"));
            m.W2 = w(STOF_NAME("W2"));
            m.bi2 = w.vector(STOF_NAME("bi2"));
            m.g2 = w.vector(STOF_NAME("g2"));
            m.b2 = w.vector(STOF_NAME("b2"));
        }
        const Launch l(hidden);
        at::Tensor x = hidden;
        PyObject* x_obj = a[1];
        int yi = 0;
        auto next_state = [&] {
            x = s.y[yi];
            x_obj = s.y_obj[yi];
            yi = (yi + 1) % s.n_y;
        };
        {
            // an index used for the first time is planned again, better, at its second use: looked up until that is done, and from
            // there on nothing needs Python
            PlanEntry plan;
            plan.decided = false;
            std::optional<Released> gil;
            for (const Layer& m : layers) {
                for (int i = 0; i < (decoder ? 2 : 1); ++i) {
                    if (!gil) {
                        plan = plan_lookup(s.ix, hidden.size(1), hidden.size(0), s.heads, s.bm, s.bn, hidden.get_device());
                        if (plan.decided) gil.emplace();
                    }
                    const Attention& w = m.a[i];
                    attention_sublayer(l, s, plan, x, w.Wqkv, w.bqkv);
                    residual_layernorm(l, fuse, s.ctx, w.Wo, w.bo, x, w.g, w.b, s.eps, s.y[yi]);
                    next_state();
                }
                gemm_core(l, x, m.W1, given(m.bi1), act, nullptr, &s.inter);
                residual_layernorm(l, fuse, s.inter, m.W2, m.bi2, x, m.g2, m.b2, s.eps, s.y[yi]);
                next_state();
            }
        }
        return same(x_obj);
    });
}

// ------------------------------------------------------------------------------------------ mask -> block index
// What a compaction in progress keeps for itself on a device: a header that its kernel leaves at zero and a record in host
// memory that the kernel writes its counts to.  A fixed number per device, made at its first compaction; a call holds one until
// it has seen its kernel's stamp, so calls from several threads and on several streams do not meet.
constexpr int NOTICES = 16;
struct NoticePool {
    char* headers = nullptr;                 // device, NOTICES x 16 bytes
    stof_mask_notice* notices = nullptr;     // pinned host memory
    unsigned long long stamp = 0;
    bool busy[NOTICES] = {};
};
NoticePool g_notices[MAX_DEVICES];           // guarded by the GIL

void cuda_ok(cudaError_t e, const char* what) {
    if (e != cudaSuccess) fail("%s failed: %s", what, cudaGetErrorString(e));
}

struct Notice {
    NoticePool& pool;
    int slot = -1;
    unsigned long long stamp = 0;
    explicit Notice(int dev) : pool(g_notices[dev]) {
        if (pool.notices == nullptr) {
            void *h = nullptr, *n = nullptr;
            cuda_ok(cudaMalloc(&h, NOTICES * 16), "cudaMalloc");
            cuda_ok(cudaMemset(h, 0, NOTICES * 16), "cudaMemset");
            cuda_ok(cudaHostAlloc(&n, NOTICES * sizeof(stof_mask_notice), cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc");
            memset(n, 0, NOTICES * sizeof(stof_mask_notice));
            cuda_ok(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
            pool.headers = static_cast<char*>(h);
            pool.notices = static_cast<stof_mask_notice*>(n);
        }
        while (slot < 0) {
            for (int i = 0; i < NOTICES && slot < 0; ++i)
                if (!pool.busy[i]) slot = i;
            if (slot < 0) {                  // sixteen other threads are waiting for theirs
                const Released gil;
                sched_yield();
            }
        }
        pool.busy[slot] = true;
        stamp = ++pool.stamp;
    }
    ~Notice() { pool.busy[slot] = false; }
    void* header() const { return pool.headers + 16 * slot; }
    stof_mask_notice* record() const { return pool.notices + slot; }
    // Polls until the kernel has written the stamp.  A stream that fails, or has nothing left to do without having written it,
    // ends the wait; the GIL is free meanwhile.
    stof_mask_notice wait(cudaStream_t stream) {
        volatile unsigned long long* at = &record()->stamp;
        cudaError_t e = cudaErrorNotReady;
        const Released gil;
        for (unsigned spins = 1; *at != stamp; ++spins) {
            if ((spins & 0x3FFF) != 0) {
                __builtin_ia32_pause();
                continue;
            }
            e = cudaStreamQuery(stream);
            if (e != cudaErrorNotReady) break;
        }
        if (*at != stamp) {
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            if (*at != stamp) fail("get_sparse_storage: the compaction did not report: %s", cudaGetErrorString(e));
        }
        __sync_synchronize();
        return *record();
    }
};

// sparse_storage(mask (batch, S, S) on the GPU, contiguous, block_m, block_n) -> the eight values of get_sparse_storage
PyObject* py_sparse_storage(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        need_args(n, 3, "sparse_storage");
        const at::Tensor& m = tensor_needed(a[0], "mask");
        need_cuda(&m);
        const int64_t bm = long_arg(a[1]), bn = long_arg(a[2]), B = m.size(0), S = m.size(2);
        if (bm <= 0 || bn <= 0 || S % bm != 0 || S % bn != 0)
            fail("get_sparse_storage: S=%lld must be a multiple of the block sizes (%lld, %lld)", static_cast<long long>(S), static_cast<long long>(bm),
                 static_cast<long long>(bn));
        const int dt = is_half(m) ? STOF_DTYPE_F16 : STOF_DTYPE_F32, s = static_cast<int>(S), ibm = static_cast<int>(bm), ibn = static_cast<int>(bn);
        const Launch l(m);
        const cudaStream_t stream = static_cast<cudaStream_t>(l.stream);
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        cuda_ok(cudaStreamIsCapturing(stream, &capturing), "cudaStreamIsCapturing");
        if (capturing != cudaStreamCaptureStatusNone) fail("get_sparse_storage: the sizes of its outputs depend on the data, so it cannot be captured");
        const int64_t rows = S / bm + 1;
        const size_t ws_bytes = api.mask_workspace_bytes(s, ibm, ibn);
        at::Tensor frp, prp, lrp, nnz, ws, fci, pci, lci, tiles;
        stof_mask_notice got;
        {
            Notice notice(m.get_device());
            const Released gil;
            frp = make({rows}, at::kInt, m);
            prp = make({rows}, at::kInt, m);
            lrp = make({rows}, at::kInt, m);
            nnz = make({}, at::kFloat, m);
            ws = make({static_cast<int64_t>(ws_bytes)}, at::kByte, m);
            call("stof_mask_classify", api.mask_classify_notify, m.data_ptr(), dt, static_cast<int>(B), s, ibm, ibn, frp.data_ptr<int>(), prp.data_ptr<int>(),
                 lrp.data_ptr<int>(), nnz.data_ptr<float>(), ws.data_ptr(), ws_bytes, notice.header(), l.status, notice.record(), notice.stamp, l.stream);
            got = notice.wait(stream);
        }
        if (got.status != 0) {
            PyObject* r = PyObject_CallFunction(g_check_status, "is", static_cast<int>(m.get_device()), "a kernel launched before this get_sparse_storage");
            if (r == nullptr) throw PythonFail{};
            Py_DECREF(r);
        }
        {
            const Released gil;
            fci = make({got.n_full}, at::kInt, m);
            pci = make({got.n_part}, at::kInt, m);
            lci = make({got.n_full + got.n_part}, at::kInt, m);
            tiles = make({got.n_part > 0 ? got.n_part : 1, bm, bn}, at::kHalf, m);
            if (got.n_part == 0) tiles.fill_(1);
            if (got.n_full + got.n_part > 0)
                call("stof_mask_fill", api.mask_fill, m.data_ptr(), dt, s, ibm, ibn, frp.data_ptr<int>(), prp.data_ptr<int>(), lrp.data_ptr<int>(),
                     fci.data_ptr<int>(), pci.data_ptr<int>(), lci.data_ptr<int>(), got.n_part > 0 ? tiles.data_ptr() : nullptr, ws.data_ptr(), ws_bytes,
                     l.stream);
        }
        const at::Tensor* out[8] = {&nnz, &frp, &fci, &prp, &pci, &tiles, &lrp, &lci};
        PyObject* tuple = PyTuple_New(8);
        for (int i = 0; i < 8; ++i) PyTuple_SET_ITEM(tuple, i, wrap(*out[i]));
        return tuple;
    });
}

// ------------------------------------------------------------------------------------------ module
// bind(library path, StofError, status_word, check_status, plan_for_call)
PyObject* py_bind(PyObject*, PyObject* args) {
    const char* path;
    PyObject *err, *status, *check_word, *plan;
    if (!PyArg_ParseTuple(args, "sOOOO", &path, &err, &status, &check_word, &plan)) return nullptr;
    void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (h == nullptr) {
        PyErr_Format(err, "cannot load %s: %s", path, dlerror());
        return nullptr;
    }
    bool ok = true;
    auto get = [&](auto& f, const char* name) {
        f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(dlsym(h, name));
        if (f == nullptr && ok) {
            PyErr_Format(err, "%s does not export %s", path, name);
            ok = false;
        }
    };
    Api x = {};
    get(x.last_error, "stof_last_error");
    get(x.mask_workspace_bytes, "stof_mask_workspace_bytes");
    get(x.mask_classify_notify, "stof_mask_classify_notify");
    get(x.mask_fill, "stof_mask_fill");
    get(x.block_attn, "stof_block_attn");
    get(x.block_attn_scheduled, "stof_block_attn_scheduled");
    get(x.gemm_bias_act, "stof_gemm_bias_act");
    get(x.gemm_ln, "stof_gemm_bias_residual_layernorm");
    get(x.layernorm, "stof_bias_residual_layernorm");
    if (!ok) return nullptr;
    api = x;
    g_error = same(err);
    g_status_word = same(status);
    g_check_status = same(check_word);
    g_plan_for_call = same(plan);
    Py_RETURN_NONE;
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, nullptr},
    FAST("gemm", py_gemm),
    FAST("gemm_ln", py_gemm_ln),
    FAST("layernorm", py_layernorm),
    FAST("attention", py_attention),
    FAST("attention_inplace", py_attention_inplace),
    FAST("merged_attention", py_merged_attention),
    FAST("stack", py_stack),
    FAST("sparse_storage", py_sparse_storage),
    {"forget", py_forget, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_stof_native", "Host path of the stof_b200 operators.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__stof_native(void) { return PyModule_Create(&module); }
