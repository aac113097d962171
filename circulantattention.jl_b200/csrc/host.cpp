// Native host path of the Python layer: shape bookkeeping, output allocation and the autograd nodes around the C ABI.
//
// A call of the public API costs one trip through here instead of a chain of Python functions, ctypes
// conversions and Python autograd nodes.  What bounds small problems is this host work, not the kernels: a
// 32 x 32 x 16 forward + backward enqueues 6 kernels that run 60 us, and the Python path took 240 us to enqueue them.
//
// Tensors are Julia-shaped column-major (H, W, C, B); the head split (src/attention.jl:44) is a reshape of
// contiguous planes, so it exists here only as numbers in the descriptor.  Every autograd node restates one of the
// reference's rrules (src/rrules.jl) as calls into the library.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/csrc/autograd/custom_function.h>
#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <nvtx3/nvToolsExt.h>

#include <cmath>
#include <mutex>
#include <optional>
#include <vector>

#include "../../include/circatt_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

namespace {

typedef c10::SmallVector<int64_t, 6> Shape;

// ---------------------------------------------------------------- errors
PyObject* g_error_class = nullptr;          // CircAttError
bool g_nvtx = false;

// Raises `cls` with `msg` on any thread (the autograd engine hands a python_error back to the caller).
[[noreturn]] void raise(PyObject* cls, const std::string& msg) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(cls, msg.c_str());
    python_error e;
    e.persist();
    throw e;
}

void check(int rc) {
    if (rc == CA_OK) return;
    raise(g_error_class, "circatt_b200 status " + std::to_string(rc) + ": " + ca_last_error());
}

void require_cuda(const Tensor& t) {
    if (!t.is_cuda())
        raise(PyExc_RuntimeError, "CirculantAttention is only CUDA compatible (no CPU path): got a tensor on " + t.device().str());
}

// ---------------------------------------------------------------- column-major tensors
bool is_colmajor(const Tensor& t) {
    int64_t expect = 1;
    const auto sz = t.sizes(), st = t.strides();
    for (size_t i = 0; i < sz.size(); ++i) {
        if (sz[i] != 1 && st[i] != expect) return false;
        expect *= sz[i];
    }
    return true;
}

Shape colmajor_strides(c10::IntArrayRef shape) {
    Shape st;
    int64_t acc = 1;
    for (int64_t n : shape) { st.push_back(acc); acc *= n; }
    return st;
}

Tensor empty_cm(c10::IntArrayRef shape, const Tensor& like, at::ScalarType dtype) {
    return at::empty_strided(shape, colmajor_strides(shape), like.options().dtype(dtype));
}

Tensor colmajor(const Tensor& t) {
    if (is_colmajor(t)) return t;
    Tensor out = empty_cm(t.sizes(), t, t.scalar_type());
    out.copy_(t);
    return out;
}

Tensor dense(const Tensor& t) {
    const auto d = t.scalar_type();
    if (d != at::kFloat && d != at::kComplexFloat && d != at::kBFloat16)
        raise(PyExc_TypeError, std::string("only Float32, ComplexF32 and (fused attention) BFloat16 are supported, got ") + c10::toString(d));
    return colmajor(t);
}

Tensor view_cm(const Tensor& t, c10::IntArrayRef shape) { return t.as_strided(shape, colmajor_strides(shape), t.storage_offset()); }

int64_t prod(c10::IntArrayRef v) {
    int64_t n = 1;
    for (int64_t x : v) n *= x;
    return n;
}

// ---------------------------------------------------------------- call context
// Device of the call, its current stream, and (per host thread) the device word in which kernels flag a wait that
// ran out.
struct StatusWords {
    std::mutex m;
    Tensor word[64];
};
StatusWords& status_words() {
    static StatusWords* w = new StatusWords;     // never destroyed: outlives the CUDA context at exit
    return *w;
}
thread_local int t_status_device = -1;

Tensor status_word(int device) {
    TORCH_CHECK(device >= 0 && device < 64, "device index out of range");
    StatusWords& s = status_words();
    Tensor w;
    {
        std::lock_guard<std::mutex> lock(s.m);
        if (!s.word[device].defined())
            s.word[device] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
        w = s.word[device];
    }
    if (t_status_device != device) {
        check(ca_status_word(w.data_ptr<int32_t>()));
        t_status_device = device;
    }
    return w;
}

struct Call {
    c10::cuda::CUDAGuard guard;
    void* stream;
    bool range;
    explicit Call(const Tensor& t, const char* name = nullptr)
        : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()), range(name && g_nvtx) {
        if (name) status_word(t.device().index());
        if (range) nvtxRangePushA(name);
    }
    ~Call() { if (range) nvtxRangePop(); }
};

Tensor scratch(size_t bytes, const Tensor& like) {
    if (!bytes) return Tensor();
    return at::empty({(int64_t)bytes}, like.options().dtype(at::kByte));
}
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }

// What a windowed kernel needs to know about a (spatial..., C, B) tensor of `nheads` heads.
struct Meta {
    int ndim;
    int64_t H, W, C, B, heads, ws;
    at::ScalarType dtype;
    int64_t Np() const { return H * W; }
    int64_t K() const { return ndim == 2 ? ws * ws : ws; }
    int64_t units() const { return heads * B; }
    ca_desc desc(int similarity = 0, int normalizer = 0, double scale = 1.0, int64_t units_ = -1) const {
        ca_desc d{};
        d.H = (int32_t)H; d.W = (int32_t)W; d.ndim = ndim;
        d.channels = (int32_t)(C / heads);
        d.units = (int32_t)(units_ < 0 ? units() : units_);
        d.ws = (int32_t)ws;
        d.dtype = dtype == at::kComplexFloat ? CA_C64 : (dtype == at::kBFloat16 ? CA_BF16 : CA_F32);
        d.similarity = similarity; d.normalizer = normalizer;
        d.scale = (float)scale;
        return d;
    }
};

Meta meta_of(const Tensor& x, int64_t ws, int64_t heads) {
    const int64_t n = x.dim();
    if (n != 3 && n != 4)
        raise(PyExc_AssertionError, "expected a (spatial..., channels, batch) array with 1 or 2 spatial dims, got " + std::to_string(n) + " dims");
    Meta m;
    m.ndim = (int)n - 2;
    m.H = x.size(0);
    m.W = n == 4 ? x.size(1) : 1;
    m.C = x.size(n - 2);
    m.B = x.size(n - 1);
    m.heads = heads;
    m.ws = ws;
    m.dtype = x.scalar_type();
    if (m.C % heads)
        raise(PyExc_AssertionError, "channels (" + std::to_string(m.C) + ") must be divisible by nheads (" + std::to_string(heads) + ")");
    return m;
}

// Descriptor of the row operators on stored values: only the spatial extents, the window and the units matter.
ca_desc nz_desc(c10::IntArrayRef spatial, int64_t ws, int64_t units, int normalizer = 0) {
    ca_desc d{};
    d.H = (int32_t)spatial[0];
    d.W = spatial.size() == 2 ? (int32_t)spatial[1] : 1;
    d.ndim = (int32_t)spatial.size();
    d.channels = 1;
    d.units = (int32_t)units;
    d.ws = (int32_t)ws;
    d.normalizer = normalizer;
    d.scale = 1.f;
    return d;
}
int64_t nz_pixels(c10::IntArrayRef spatial) { return prod(spatial); }

bool tracked(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// ---------------------------------------------------------------- similarity
// Values of shape (Np*K, heads, B).
Tensor similarity_raw(int64_t kind, const Tensor& x_, const Tensor& y_, int64_t ws, double scale, int64_t heads) {
    require_cuda(x_);
    require_cuda(y_);
    const Tensor x = dense(x_), y = dense(y_);
    const Meta m = meta_of(x, ws, heads);
    Call call(x);
    Tensor nz = empty_cm({m.Np() * m.K(), heads, m.B}, x, at::kFloat);
    const ca_desc d = m.desc((int)kind, 0, scale);
    const Tensor w = scratch(ca_operator_workspace(&d), x);
    check(ca_similarity(&d, ptr(x), ptr(y), fptr(nz), ptr(w), call.stream));
    return nz;
}

std::tuple<Tensor, Tensor> similarity_bwd_raw(int64_t kind, const Tensor& x_, const Tensor& y_, int64_t ws, const Tensor& dS_,
                                              double scale, int64_t heads, bool need_x = true, bool need_y = true) {
    const Tensor x = dense(x_), y = dense(y_), dS = colmajor(dS_);
    const Meta m = meta_of(x, ws, heads);
    Call call(x);
    Tensor dx, dy;
    if (need_x) dx = empty_cm(x.sizes(), x, x.scalar_type());
    if (need_y) dy = empty_cm(y.sizes(), y, y.scalar_type());
    const ca_desc d = m.desc((int)kind, 0, scale);
    const Tensor w = scratch(ca_operator_workspace(&d), x);
    check(ca_similarity_bwd(&d, ptr(x), ptr(y), fptr(dS), ptr(dx), ptr(dy), ptr(w), call.stream));
    return {dx, dy};
}

// circulant_similarity and its rrules (src/similarity.jl:138-142, src/rrules.jl:1-32).
struct SimilarityFn : public Function<SimilarityFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& y, int64_t kind, int64_t ws, int64_t heads) {
        ctx->save_for_backward({x, y});
        ctx->saved_data["kind"] = kind;
        ctx->saved_data["ws"] = ws;
        ctx->saved_data["heads"] = heads;
        return similarity_raw(kind, x, y, ws, 1.0, heads);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        auto [dx, dy] = similarity_bwd_raw(ctx->saved_data["kind"].toInt(), s[0], s[1], ctx->saved_data["ws"].toInt(), g[0], 1.0,
                                           ctx->saved_data["heads"].toInt(), ctx->needs_input_grad(0), ctx->needs_input_grad(1));
        return {dx, dy, Tensor(), Tensor(), Tensor()};
    }
};

Tensor similarity(const Tensor& x, const Tensor& y, int64_t kind, int64_t ws, int64_t heads) {
    if (!tracked({&x, &y})) return similarity_raw(kind, x, y, ws, 1.0, heads);
    return SimilarityFn::apply(x, y, kind, ws, heads);
}

// ---------------------------------------------------------------- row normaliser
std::tuple<Tensor, Tensor> normalize_raw(const Tensor& nz_, const std::vector<int64_t>& spatial, int64_t ws, int64_t normalizer,
                                         const std::optional<Tensor>& out_, bool want_stats) {
    require_cuda(nz_);
    const Tensor nz = colmajor(nz_);
    const int64_t units = nz.numel() / nz.size(0);
    Call call(nz);
    Tensor out = out_ ? *out_ : empty_cm(nz.sizes(), nz, at::kFloat), stats;
    if (want_stats) stats = empty_cm({nz_pixels(spatial), units}, nz, at::kFloat);
    const ca_desc d = nz_desc(spatial, ws, units, (int)normalizer);
    check(ca_row_normalize(&d, fptr(nz), fptr(out), fptr(stats), call.stream));
    return {out, stats};
}

Tensor normalize_bwd_raw(const Tensor& p_, const Tensor& dp_, const std::vector<int64_t>& spatial, int64_t ws, int64_t normalizer) {
    const Tensor p = colmajor(p_), dp = colmajor(dp_);
    Call call(p);
    Tensor ds = empty_cm(p.sizes(), p, at::kFloat);
    const ca_desc d = nz_desc(spatial, ws, p.numel() / p.size(0), (int)normalizer);
    check(ca_row_normalize_bwd(&d, fptr(p), fptr(dp), fptr(ds), call.stream));
    return ds;
}

// NNlib.softmax(::Circulant) and its rrule (src/similarity.jl:113-126, src/rrules.jl:42-56).
struct NormalizeFn : public Function<NormalizeFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& nz, std::vector<int64_t> spatial, int64_t ws, int64_t normalizer) {
        Tensor p = std::get<0>(normalize_raw(nz, spatial, ws, normalizer, std::nullopt, false));
        ctx->save_for_backward({p});
        ctx->saved_data["spatial"] = spatial;
        ctx->saved_data["ws"] = ws;
        ctx->saved_data["normalizer"] = normalizer;
        return p;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        return {normalize_bwd_raw(s[0], g[0], ctx->saved_data["spatial"].toIntVector(), ctx->saved_data["ws"].toInt(),
                                  ctx->saved_data["normalizer"].toInt()), Tensor(), Tensor(), Tensor()};
    }
};

Tensor normalize(const Tensor& nz, const std::vector<int64_t>& spatial, int64_t ws, int64_t normalizer) {
    if (!tracked({&nz})) return std::get<0>(normalize_raw(nz, spatial, ws, normalizer, std::nullopt, false));
    return NormalizeFn::apply(nz, spatial, ws, normalizer);
}

// ---------------------------------------------------------------- adjacency
// softmax o circulant_similarity and the composition of their rrules (src/similarity.jl:157-161, src/rrules.jl:1-56) as one
// node instead of two (a host-bound graph of two adjacencies, 96 x 80 x 32 x 2, ws 9, with every gradient: 276 -> 254 us).
Tensor adjacency_raw(const Tensor& x, const Tensor& y, int64_t kind, int64_t ws, int64_t heads, int64_t normalizer) {
    const Tensor s = similarity_raw(kind, x, y, ws, 1.0, heads);          // checks x and y
    const std::vector<int64_t> spatial(x.sizes().begin(), x.sizes().end() - 2);
    return std::get<0>(normalize_raw(s, spatial, ws, normalizer, std::nullopt, false));
}

struct AdjacencyFn : public Function<AdjacencyFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& y, int64_t kind, int64_t ws, int64_t heads, int64_t normalizer) {
        Tensor p = adjacency_raw(x, y, kind, ws, heads, normalizer);
        ctx->save_for_backward({x, y, p});
        ctx->saved_data["kind"] = kind;
        ctx->saved_data["ws"] = ws;
        ctx->saved_data["heads"] = heads;
        ctx->saved_data["normalizer"] = normalizer;
        return p;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const Tensor &x = s[0], &y = s[1];
        const int64_t ws = ctx->saved_data["ws"].toInt();
        const std::vector<int64_t> spatial(x.sizes().begin(), x.sizes().end() - 2);
        const Tensor ds = normalize_bwd_raw(s[2], g[0], spatial, ws, ctx->saved_data["normalizer"].toInt());
        auto [dx, dy] = similarity_bwd_raw(ctx->saved_data["kind"].toInt(), x, y, ws, ds, 1.0, ctx->saved_data["heads"].toInt(),
                                           ctx->needs_input_grad(0), ctx->needs_input_grad(1));
        return {dx, dy, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

Tensor adjacency(const Tensor& x, const Tensor& y, int64_t kind, int64_t ws, int64_t heads, int64_t normalizer) {
    if (!tracked({&x, &y})) return adjacency_raw(x, y, kind, ws, heads, normalizer);
    return AdjacencyFn::apply(x, y, kind, ws, heads, normalizer);
}

// ---------------------------------------------------------------- apply
// A (x) v or A^T (x) v.  nz: (Np*K, batch...); v: (spatial..., C, B) of `heads` heads.  Where the units of A are
// broadcast over those of v or the other way round, the result has the larger number of units.
Tensor apply_raw(const Tensor& nz_, const Tensor& v_, int64_t ws, bool transpose, int64_t heads, const std::optional<Tensor>& out_) {
    require_cuda(nz_);
    require_cuda(v_);
    const Tensor nz = colmajor(nz_), v = dense(v_);
    const Meta m = meta_of(v, ws, heads);
    const int64_t ua = nz.numel() / nz.size(0), uv = m.units(), units = std::max(ua, uv);
    if ((ua != 1 && ua != units) || (uv != 1 && uv != units))
        raise(PyExc_AssertionError, "batch dims of A (" + std::to_string(ua) + ") and of x (" + std::to_string(uv) + ") do not broadcast");
    if (nz.size(0) != m.Np() * m.K())
        raise(PyExc_AssertionError, "A has " + std::to_string(nz.size(0)) + " stored entries per batch, x needs " + std::to_string(m.Np() * m.K()));
    Call call(v);
    Tensor out;
    if (out_) {
        out = *out_;
    } else if (units == uv) {
        out = empty_cm(v.sizes(), v, v.scalar_type());
    } else {
        Shape sh(v.sizes().begin(), v.sizes().end());
        sh[sh.size() - 2] = m.C / heads;
        sh[sh.size() - 1] = units;
        out = empty_cm(sh, v, v.scalar_type());
    }
    const ca_desc d = m.desc(0, 0, 1.0, units);
    const Tensor w = scratch(ca_operator_workspace(&d), v);
    check(ca_apply(&d, fptr(nz), ptr(v), ptr(out), transpose, ua == 1 && units > 1, uv == 1 && units > 1, ptr(w), call.stream));
    return out;
}

// A (x) x, A^T (x) x and their rrules (src/attention.jl:53-80, src/rrules.jl:58-88).
struct ApplyFn : public Function<ApplyFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& nz, const Tensor& x, int64_t ws, bool transpose, int64_t heads) {
        ctx->save_for_backward({nz, x});
        ctx->saved_data["ws"] = ws;
        ctx->saved_data["transpose"] = transpose;
        ctx->saved_data["heads"] = heads;
        return apply_raw(nz, x, ws, transpose, heads, std::nullopt);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const Tensor &nz = s[0], &x = s[1], &dc = g[0];
        const int64_t ws = ctx->saved_data["ws"].toInt(), heads = ctx->saved_data["heads"].toInt();
        const bool transpose = ctx->saved_data["transpose"].toBool();
        if (nz.numel() / nz.size(0) != heads * x.size(x.dim() - 1))
            raise(PyExc_NotImplementedError, "pullback of a batch-broadcast apply is not defined by the reference");
        Tensor dA, db;
        if (ctx->needs_input_grad(0)) {
            const Tensor d = transpose ? similarity_raw(CA_DOT, x, dc, ws, 1.0, heads) : similarity_raw(CA_DOT, dc, x, ws, 1.0, heads);
            dA = view_cm(d, nz.sizes());
        }
        if (ctx->needs_input_grad(1)) db = apply_raw(nz, dc, ws, !transpose, heads, std::nullopt);
        return {dA, db, Tensor(), Tensor(), Tensor()};
    }
};

Tensor apply(const Tensor& nz, const Tensor& x, int64_t ws, bool transpose, int64_t heads) {
    if (!tracked({&nz, &x})) return apply_raw(nz, x, ws, transpose, heads, std::nullopt);
    return ApplyFn::apply(nz, x, ws, transpose, heads);
}

// ---------------------------------------------------------------- fused attention
struct FwdOut { Tensor y, nz, stats, workspace; };

FwdOut attention_fwd_raw(const Tensor& q, const Tensor& k, const Tensor& v, int64_t kind, int64_t ws, int64_t normalizer,
                         bool want_a, double scale, int64_t heads) {
    const Meta m = meta_of(q, ws, heads);
    Call call(q, "circatt.fwd");
    const ca_desc d = m.desc((int)kind, (int)normalizer, scale);
    FwdOut o;
    o.y = empty_cm(q.sizes(), q, q.scalar_type());
    if (want_a) o.nz = empty_cm({m.Np() * m.K(), heads, m.B}, q, at::kFloat);
    o.stats = empty_cm({m.Np(), m.units()}, q, at::kFloat);
    o.workspace = scratch(ca_attention_fwd_workspace(&d, want_a), q);
    check(ca_attention_fwd(&d, ptr(q), ptr(k), ptr(v), ptr(o.y), fptr(o.nz), fptr(o.stats), ptr(o.workspace), call.stream));
    return o;
}

// circulant_(mh_)attention with a direct pullback equal to the composition of the reference's rrules
// (src/rrules.jl:1-72).  The forward's workspace (the packed copy of k and v) is kept for the softmax pullback, like
// the intermediates that the reference's pullback closures capture (src/rrules.jl:44-55).
struct AttentionFn : public Function<AttentionFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, int64_t kind,
                                 int64_t ws, int64_t normalizer, bool want_a, double scale, int64_t heads) {
        const Tensor q = dense(q_), k = dense(k_), v = dense(v_);
        FwdOut o = attention_fwd_raw(q, k, v, kind, ws, normalizer, want_a, scale, heads);
        ctx->set_materialize_grads(false);            // an unused A arrives as undefined, not as zeros, in backward
        ctx->save_for_backward({q, k, v, o.y, o.stats, o.nz, normalizer == CA_SOFTMAX ? o.workspace : Tensor()});
        ctx->saved_data["kind"] = kind;
        ctx->saved_data["ws"] = ws;
        ctx->saved_data["normalizer"] = normalizer;
        ctx->saved_data["scale"] = scale;
        ctx->saved_data["heads"] = heads;
        return want_a ? variable_list{o.y, o.nz} : variable_list{o.y};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const Tensor &q = s[0], &k = s[1], &v = s[2], &y = s[3], &stats = s[4], &nz = s[5], &fws = s[6];
        const Meta m = meta_of(q, ctx->saved_data["ws"].toInt(), ctx->saved_data["heads"].toInt());
        const Tensor dA = g.size() > 1 && g[1].defined() ? colmajor(g[1]) : Tensor();
        Call call(q, "circatt.bwd");
        Tensor dy;
        if (g[0].defined()) dy = dense(g[0]);
        else { dy = empty_cm(q.sizes(), q, q.scalar_type()); dy.zero_(); }
        const ca_desc d = m.desc((int)ctx->saved_data["kind"].toInt(), (int)ctx->saved_data["normalizer"].toInt(),
                                 ctx->saved_data["scale"].toDouble());
        Tensor dq = empty_cm(q.sizes(), q, q.scalar_type()), dk = empty_cm(q.sizes(), q, q.scalar_type()),
               dv = empty_cm(q.sizes(), q, q.scalar_type());
        const Tensor w = scratch(ca_attention_bwd_workspace(&d, dA.defined()), q);
        check(ca_attention_bwd(&d, ptr(q), ptr(k), ptr(v), ptr(y), ptr(dy), fptr(stats), fptr(nz), fptr(dA), ptr(dq), ptr(dk), ptr(dv),
                               ptr(w), ptr(fws), call.stream));
        return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// (y, values of A or None)
std::tuple<Tensor, std::optional<Tensor>> attention(const Tensor& q, const Tensor& k, const Tensor& v, int64_t kind, int64_t ws,
                                                    int64_t normalizer, bool want_a, std::optional<double> scale_, int64_t heads) {
    require_cuda(q);
    require_cuda(k);
    require_cuda(v);
    const double scale = scale_ ? *scale_ : 1.0 / std::sqrt((double)(q.size(q.dim() - 2) / heads));
    if (!tracked({&q, &k, &v})) {
        FwdOut o = attention_fwd_raw(dense(q), dense(k), dense(v), kind, ws, normalizer, want_a, scale, heads);
        return {o.y, want_a ? std::optional<Tensor>(o.nz) : std::nullopt};
    }
    variable_list o = AttentionFn::apply(q, k, v, kind, ws, normalizer, want_a, scale, heads);
    return {o[0], want_a ? std::optional<Tensor>(o[1]) : std::nullopt};
}

// ---------------------------------------------------------------- algebra on values
Tensor axpby_raw(double alpha, const Tensor& x_, double beta, const std::optional<Tensor>& y_) {
    require_cuda(x_);
    if (y_) require_cuda(*y_);
    const Tensor x = colmajor(x_), y = y_ ? colmajor(*y_) : Tensor();
    Call call(x);
    Tensor out = empty_cm(x.sizes(), x, at::kFloat);
    check(ca_axpby(x.numel(), (float)alpha, fptr(x), (float)beta, fptr(y), fptr(out), call.stream));
    return out;
}

struct AxpbyFn : public Function<AxpbyFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& y, double alpha, double beta) {
        ctx->saved_data["alpha"] = alpha;
        ctx->saved_data["beta"] = beta;
        ctx->saved_data["two"] = y.has_value();
        return axpby_raw(alpha, x, beta, y);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        Tensor gx, gy;
        auto times = [&](double c) { return c == 1.0 ? g[0] : axpby_raw(c, g[0], 0.0, std::nullopt); };
        if (ctx->needs_input_grad(0)) gx = times(ctx->saved_data["alpha"].toDouble());
        if (ctx->saved_data["two"].toBool() && ctx->needs_input_grad(1)) gy = times(ctx->saved_data["beta"].toDouble());
        return {gx, gy, Tensor(), Tensor()};
    }
};

Tensor axpby(const Tensor& x, const std::optional<Tensor>& y, double alpha, double beta) {
    if (!tracked({&x}) && !(y && tracked({&*y}))) return axpby_raw(alpha, x, beta, y);
    return AxpbyFn::apply(x, y, alpha, beta);
}

struct Batch2 { int64_t b[2] = {1, 1}; };
Batch2 batch_of(c10::IntArrayRef sizes, size_t first) {
    if (sizes.size() > first + 2) raise(PyExc_NotImplementedError, "at most two batch dims (heads, batch) are supported");
    Batch2 r;
    for (size_t i = first; i < sizes.size(); ++i) r.b[i - first] = sizes[i];
    return r;
}

// nz (inner, a...) times c (c...) with Julia-style extent-1 broadcasting.
Tensor scale_batch_raw(const Tensor& c_, const Tensor& nz_) {
    require_cuda(c_);
    require_cuda(nz_);
    const Tensor c = colmajor(c_), nz = colmajor(nz_);
    const Batch2 a = batch_of(nz.sizes(), 1), cb = batch_of(c.sizes(), 0);
    const int64_t o1 = std::max(a.b[0], cb.b[0]), o2 = std::max(a.b[1], cb.b[1]);
    const int64_t nb = std::max(nz.dim() - 1, c.dim());
    Shape sh{nz.size(0)};
    if (nb > 0) sh.push_back(o1);
    if (nb > 1) sh.push_back(o2);
    Call call(nz);
    Tensor out = empty_cm(sh, nz, at::kFloat);
    check(ca_scale_batch(nz.size(0), (int32_t)o1, (int32_t)o2, fptr(nz), (int32_t)a.b[0], (int32_t)a.b[1], fptr(c),
                         (int32_t)cb.b[0], (int32_t)cb.b[1], fptr(out), call.stream));
    return out;
}

// per-slice sum_n x*y (no y: sum of x); x, y: (inner, b...) broadcasting -> (b...)
Tensor dot_batch_raw(const Tensor& x_, const std::optional<Tensor>& y_) {
    require_cuda(x_);
    if (y_) require_cuda(*y_);
    const Tensor x = colmajor(x_), y = y_ ? colmajor(*y_) : Tensor();
    const Batch2 xb = batch_of(x.sizes(), 1), yb = y_ ? batch_of(y.sizes(), 1) : Batch2();
    const int64_t o1 = std::max(xb.b[0], yb.b[0]), o2 = std::max(xb.b[1], yb.b[1]);
    const int64_t nb = std::max(x.dim(), y_ ? y.dim() : 0) - 1;
    Shape sh;
    if (nb == 0) sh.push_back(1);
    if (nb > 0) sh.push_back(o1);
    if (nb > 1) sh.push_back(o2);
    Call call(x);
    Tensor out = empty_cm(sh, x, at::kFloat);
    check(ca_dot_batch(x.size(0), (int32_t)o1, (int32_t)o2, fptr(x), (int32_t)xb.b[0], (int32_t)xb.b[1], fptr(y), (int32_t)yb.b[0],
                       (int32_t)yb.b[1], fptr(out), call.stream));
    return out;
}

Tensor sum_batch_raw(const Tensor& nz_, bool sum1, bool sum2) {
    require_cuda(nz_);
    const Tensor nz = colmajor(nz_);
    const Batch2 b = batch_of(nz.sizes(), 1);
    Shape sh{nz.size(0)};
    if (nz.dim() > 1) sh.push_back(sum1 ? 1 : b.b[0]);
    if (nz.dim() > 2) sh.push_back(sum2 ? 1 : b.b[1]);
    Call call(nz);
    Tensor out = empty_cm(sh, nz, at::kFloat);
    check(ca_sum_batch(nz.size(0), (int32_t)b.b[0], (int32_t)b.b[1], sum1, sum2, fptr(nz), fptr(out), call.stream));
    return out;
}

// scale(c, A) and its pullback (src/array.jl:179-186, src/rrules.jl:97-114).
struct ScaleFn : public Function<ScaleFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& c, const Tensor& nz) {
        ctx->save_for_backward({c, nz});
        return scale_batch_raw(c, nz);
    }
    // sums `full` (inner, o1, o2) over the batch dims in which `b` was broadcast
    static Tensor reduce(const Tensor& full, const Batch2& b, c10::IntArrayRef shape) {
        const bool s1 = full.dim() > 1 && b.b[0] == 1 && full.size(1) > 1;
        const bool s2 = full.dim() > 2 && b.b[1] == 1 && full.size(2) > 1;
        return view_cm(s1 || s2 ? sum_batch_raw(full, s1, s2) : full, shape);
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const Tensor &c = s[0], &nz = s[1];
        Tensor dc, dA;
        if (ctx->needs_input_grad(0)) {
            const Tensor d = dot_batch_raw(g[0], nz);                         // (o1, o2): per-slice sum dB*A
            Shape sh{1};
            for (int64_t n : d.sizes()) sh.push_back(n);
            dc = reduce(view_cm(d, sh), batch_of(c.sizes(), 0), c.sizes());
        }
        if (ctx->needs_input_grad(1)) dA = reduce(scale_batch_raw(c, g[0]), batch_of(nz.sizes(), 1), nz.sizes());
        return {dc, dA};
    }
};

Tensor scale_batch(const Tensor& c, const Tensor& nz) {
    if (!tracked({&c, &nz})) return scale_batch_raw(c, nz);
    return ScaleFn::apply(c, nz);
}

Tensor sum_axis_raw(const Tensor& nz_, const std::vector<int64_t>& spatial, int64_t ws, bool rows) {
    require_cuda(nz_);
    const Tensor nz = colmajor(nz_);
    const int64_t Np = nz_pixels(spatial);
    Shape sh{rows ? Np : 1, rows ? 1 : Np};
    for (int64_t i = 1; i < nz.dim(); ++i) sh.push_back(nz.size(i));
    Call call(nz);
    Tensor out = empty_cm(sh, nz, at::kFloat);
    const ca_desc d = nz_desc(spatial, ws, nz.numel() / nz.size(0));
    check((rows ? ca_sum_rows : ca_sum_cols)(&d, fptr(nz), fptr(out), call.stream));
    return out;
}

// Julia `reshape` (column-major): a view where `t` is column-major.
Tensor reshape(const Tensor& t_, std::vector<int64_t> shape) {
    int64_t known = 1, hole = -1;
    for (size_t i = 0; i < shape.size(); ++i) {
        if (shape[i] == -1 && hole < 0) hole = (int64_t)i;
        else known *= shape[i];
    }
    if (hole >= 0) shape[hole] = t_.numel() / std::max<int64_t>(known, 1);
    if (!tracked({&t_})) return view_cm(colmajor(t_), shape);
    Shape rev, target;
    for (int64_t i = t_.dim() - 1; i >= 0; --i) rev.push_back(i);
    for (size_t i = shape.size(); i-- > 0;) target.push_back(shape[i]);
    Tensor flat = t_.permute(rev).contiguous().view(target);
    rev.clear();
    for (int64_t i = (int64_t)shape.size() - 1; i >= 0; --i) rev.push_back(i);
    return flat.permute(rev);
}

}  // namespace

PYBIND11_MODULE(_circatt_host, m) {
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (python_error& e) {
            e.restore();
        }
    });
    using release = py::call_guard<py::gil_scoped_release>;
    m.def("set_error_class", [](py::object cls) { Py_XDECREF(g_error_class); g_error_class = cls.release().ptr(); });
    m.def("enable_nvtx", [](bool flag) { const bool old = g_nvtx; g_nvtx = flag; return old; });
    m.def("status_word", &status_word, release());
    m.def("has_status_word", [](int device) {
        std::lock_guard<std::mutex> lock(status_words().m);
        return device >= 0 && device < 64 && status_words().word[device].defined();
    });
    m.def("attention", &attention, release());
    m.def("similarity", &similarity, release());
    m.def("adjacency", &adjacency, release());
    m.def("similarity_raw", [](int64_t kind, const Tensor& x, const Tensor& y, int64_t ws, double scale) {
        const Tensor nz = similarity_raw(kind, x, y, ws, scale, 1);
        return view_cm(nz, {nz.size(0), nz.size(2)});
    }, py::arg("kind"), py::arg("x"), py::arg("y"), py::arg("ws"), py::arg("scale") = 1.0, release());
    m.def("similarity_bwd_raw", [](int64_t kind, const Tensor& x, const Tensor& y, int64_t ws, const Tensor& dS, double scale) {
        return similarity_bwd_raw(kind, x, y, ws, dS, scale, 1);
    }, py::arg("kind"), py::arg("x"), py::arg("y"), py::arg("ws"), py::arg("dS"), py::arg("scale") = 1.0, release());
    m.def("normalize", &normalize, release());
    m.def("normalize_raw", &normalize_raw, release());
    m.def("normalize_bwd_raw", &normalize_bwd_raw, release());
    m.def("apply", &apply, release());
    m.def("apply_raw", &apply_raw, release());
    m.def("axpby", &axpby, release());
    m.def("axpby_raw", &axpby_raw, release());
    m.def("scale_batch", &scale_batch, release());
    m.def("scale_batch_raw", &scale_batch_raw, release());
    m.def("dot_batch", &dot_batch_raw, release());
    m.def("sum_batch", &sum_batch_raw, release());
    m.def("sum_axis", &sum_axis_raw, release());
    m.def("reshape", &reshape, release());
}
