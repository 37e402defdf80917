// The package's autograd nodes in C++: the fused operator, the fused operator on a packed projection output, the
// drop-in pair, the attention layer, and the transformer block. They call the C ABI (include/na1d_b200.h) and nothing else of their own.
//
// A forward and backward of the operator through a Python autograd.Function cost 140 to 170 us of host time (argument
// conversions through ctypes, and a backward that needs the interpreter on the autograd thread) while its kernels take 5 to
// 60 us at the usual sizes: the host bound them all.
//
// Every entry returns None where the call is anything but plain eager tensors of the forms the kernels take -- wrapped
// tensors, dispatch modes, tracing, functorch transforms, forward-mode derivatives, other types, layouts, sizes -- and the
// caller goes on to the Python route, which supports or refuses it as it always has.
#include <torch/extension.h>

#include <cublasLt.h>
#include <unordered_map>

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/tunable/Tunable.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "../../include/na1d_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// Raises the package's own exception; also from a thread that does not hold the interpreter lock.
[[noreturn]] void raise_status(int status, const char* where) {
    py::gil_scoped_acquire gil;
    py::object cls = py::module_::import("pcf_nat_b200._lib").attr("Na1dError");
    py::object exc = cls(status, where);
    PyErr_SetObject(cls.ptr(), exc.ptr());
    throw py::error_already_set();
}
inline void check(int status, const char* where) {
    if (status != 0) raise_status(status, where);
}
inline void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }
inline int code(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? NA1D_BF16 : NA1D_FP16; }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }
inline Tensor empty_f32(at::IntArrayRef shape, const Tensor& like) { return at::empty(shape, like.options().dtype(at::kFloat)); }

inline Tensor zeros_f32(at::IntArrayRef shape, const Tensor& like) {
    const Tensor t = empty_f32(shape, like);
    check(na1d_zero(ptr(t), t.numel() * 4, stream()), "na1d_zero");
    return t;
}

// ---------------------------------------------------------------- library products
// y (rows, N) = x (rows, K) w^T + b with w (N, K), or x w with w (K, N), dense and 16-bit, sums in fp32: the library product that at::addmm
// and at::mm run, without their work for each call (13 to 16 us of host time, 5 here). What the library proposes for sizes, types and
// alignments is kept under exactly those, for each host thread by itself, 256 of them at most.
struct ProductKey {
    int64_t rows, N, K, ldw, ldc;   // ldc: 0 without an addend
    int32_t kind, align;   // device, type, orientation, bias; the operands' alignments
    bool operator==(const ProductKey& o) const {
        return rows == o.rows && N == o.N && K == o.K && ldw == o.ldw && ldc == o.ldc && kind == o.kind && align == o.align;
    }
};
struct ProductKeyHash {
    size_t operator()(const ProductKey& k) const {
        size_t h = 1469598103934665603ull;
        for (size_t v : {(size_t)k.rows, (size_t)k.N, (size_t)k.K, (size_t)k.ldw, (size_t)k.ldc, (size_t)k.kind, (size_t)k.align}) h = (h ^ v) * 1099511628211ull;
        return h ^ (h >> 29);
    }
};
struct ProductPlan {
    cublasLtMatmulDescOpaque_t desc;
    cublasLtMatrixLayoutOpaque_t w, x, y, c;
    cublasLtMatmulAlgo_t algo;
    bool usable;
};
int32_t alignment(const void* p) {   // 16, 32, .. 256 bytes as 0 .. 4; -1: less
    const auto a = reinterpret_cast<uintptr_t>(p);
    int32_t n = -1;
    for (uintptr_t b = 16; b <= 256 && (a & (b - 1)) == 0; b *= 2) ++n;
    return n;
}
bool plan_product(ProductPlan& p, const ProductKey& k, cublasLtHandle_t handle, cudaDataType_t type, bool w_transposed, bool bias, const int32_t (&align)[4]) {
    p.usable = false;
    // the library counts columns first: y^T (N, rows) = op(w) x^T
    const cublasOperation_t op = w_transposed ? CUBLAS_OP_N : CUBLAS_OP_T;
    const cublasLtEpilogue_t epilogue = CUBLASLT_EPILOGUE_BIAS;
    const uint32_t reductions = CUBLASLT_REDUCTION_SCHEME_NONE | CUBLASLT_REDUCTION_SCHEME_COMPUTE_TYPE;   // partial sums stay fp32
    const size_t workspace = at::cuda::getCUDABlasLtWorkspaceSize();
    cublasLtMatmulPreferenceOpaque_t pref;
    if (cublasLtMatmulDescInit(&p.desc, CUBLAS_COMPUTE_32F, CUDA_R_32F) || cublasLtMatmulDescSetAttribute(&p.desc, CUBLASLT_MATMUL_DESC_TRANSA, &op, sizeof op) ||
        cublasLtMatrixLayoutInit(&p.w, type, w_transposed ? k.N : k.K, w_transposed ? k.K : k.N, k.ldw) ||
        cublasLtMatrixLayoutInit(&p.x, type, k.K, k.rows, k.K) || cublasLtMatrixLayoutInit(&p.y, type, k.N, k.rows, k.N) ||
        cublasLtMatrixLayoutInit(&p.c, type, k.N, k.rows, k.ldc ? k.ldc : k.N) || cublasLtMatmulPreferenceInit(&pref) ||
        cublasLtMatmulPreferenceSetAttribute(&pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &workspace, sizeof workspace) ||
        cublasLtMatmulPreferenceSetAttribute(&pref, CUBLASLT_MATMUL_PREF_REDUCTION_SCHEME_MASK, &reductions, sizeof reductions))
        return false;
    if (bias && (cublasLtMatmulDescSetAttribute(&p.desc, CUBLASLT_MATMUL_DESC_EPILOGUE, &epilogue, sizeof epilogue) ||
                 cublasLtMatmulDescSetAttribute(&p.desc, CUBLASLT_MATMUL_DESC_BIAS_DATA_TYPE, &type, sizeof type)))
        return false;
    const cublasLtMatmulPreferenceAttributes_t which[3] = {CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES,
                                                           CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES};
    for (int i = 0; i < 3; ++i) {
        const uint32_t bytes = 16u << align[i];
        if (cublasLtMatmulPreferenceSetAttribute(&pref, which[i], &bytes, sizeof bytes)) return false;
    }
    cublasLtMatmulHeuristicResult_t found = {};
    int n = 0;
    if (cublasLtMatmulAlgoGetHeuristic(handle, &p.desc, &p.w, &p.x, &p.c, &p.y, &pref, 1, &found, &n) || n < 1) return false;
    p.algo = found.algo;
    p.usable = true;
    return true;
}
// Settings of the framework's that say how its products run (a preferred library, tuned products, deterministic algorithms, 16-bit sums, no
// split sums) are its own operations' to follow.
bool default_products(at::ScalarType type) {
    auto& ctx = at::globalContext();
    const auto backend = ctx.blasPreferredBackend();
    const auto sums = type == at::kBFloat16 ? ctx.allowBF16ReductionCuBLAS() : ctx.allowFP16ReductionCuBLAS();
    return (backend == at::BlasBackend::Default || backend == at::BlasBackend::Cublas) && !ctx.deterministicAlgorithms() &&
           sums != at::CuBLASReductionOption::DisallowReducedPrecisionDisallowSplitK && !ctx.allowFP16AccumulationCuBLAS() &&
           !at::cuda::tunable::getTuningContext()->IsTunableOpEnabled();
}
// `add`, (rows, N): added before the result is rounded. It and w may be column slices of wider matrices.
Tensor product(const Tensor& x, const Tensor& w, const Tensor& b, bool w_transposed, const Tensor& add = Tensor()) {
    const int64_t rows = x.size(0), K = x.size(1), N = w.size(w_transposed ? 1 : 0);
    Tensor y = at::empty({rows, N}, x.options());
    const bool bias = b.defined(), sum = add.defined();
    const int32_t align[4] = {alignment(ptr(w)), alignment(ptr(x)), sum ? std::min(alignment(ptr(add)), alignment(ptr(y))) : alignment(ptr(y)),
                              bias ? alignment(ptr(b)) : 4};
    auto slice = [](const Tensor& t) { return t.stride(1) == 1 && t.stride(0) >= t.size(1) && t.stride(0) % 8 == 0; };
    const bool dense = x.is_contiguous() && slice(w) && (!sum || slice(add)) && K % 8 == 0 && N % 8 == 0 && rows <= INT32_MAX && align[0] >= 0 && align[1] >= 0 && align[2] >= 0 && align[3] >= 0;
    if (dense && default_products(x.scalar_type())) {
        static thread_local std::unordered_map<ProductKey, ProductPlan, ProductKeyHash> plans;
        const cudaDataType_t type = x.scalar_type() == at::kBFloat16 ? CUDA_R_16BF : CUDA_R_16F;
        const ProductKey key{rows, N, K, w.stride(0), sum ? add.stride(0) : 0, (int32_t)(x.get_device() * 8 + code(x) * 4 + w_transposed * 2 + bias), align[0] | align[1] << 4 | align[2] << 8};
        const cublasLtHandle_t handle = at::cuda::getCurrentCUDABlasLtHandle();
        auto it = plans.find(key);
        if (it == plans.end()) {
            if (plans.size() >= 256) plans.clear();
            it = plans.emplace(key, ProductPlan()).first;
            plan_product(it->second, key, handle, type, w_transposed, bias, align);
        }
        ProductPlan& p = it->second;
        const void* bp = ptr(b);
        const float one = 1.f, beta = sum ? 1.f : 0.f;
        if (p.usable && !(bias && cublasLtMatmulDescSetAttribute(&p.desc, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bp, sizeof bp)) &&
            cublasLtMatmul(handle, &p.desc, &one, ptr(w), &p.w, ptr(x), &p.x, &beta, sum ? ptr(add) : ptr(y), &p.c, ptr(y), &p.y, &p.algo, at::cuda::getCUDABlasLtWorkspace(),
                           at::cuda::getCUDABlasLtWorkspaceSize(), at::cuda::getCurrentCUDAStream().stream()) == CUBLAS_STATUS_SUCCESS)
            return y;
    }
    if (sum) return at::add(at::mm(x, w_transposed ? w : w.t()), add);
    if (!bias) return at::mm(x, w_transposed ? w : w.t());
    return at::addmm(b, x, w_transposed ? w : w.t());
}

bool eager_mode() {
    return c10::impl::TorchDispatchModeTLS::stack_len() == 0 && !torch::jit::tracer::isTracing() &&
           !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}
bool plain(const Tensor& t) {
    return t.defined() && t.has_storage() && t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has(c10::DispatchKey::Python) &&
           !t._is_zerotensor() && !t.is_neg() && !t._fw_grad(0).defined();
}
bool plain16(const Tensor& t) { return plain(t) && (t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf); }
// bias and valid lengths as the kernels want them; false: not a form this route takes
bool prepare_rpb(const OptTensor& rpb, int64_t n, const Tensor& like) {
    return !rpb || !rpb->defined() || (plain(*rpb) && rpb->device() == like.device() && rpb->numel() == n && at::isFloatingType(rpb->scalar_type()));
}
Tensor rpb32(const OptTensor& rpb) {
    if (!rpb || !rpb->defined()) return Tensor();
    const Tensor r = rpb->detach();
    return (r.scalar_type() == at::kFloat ? r : r.to(at::kFloat)).contiguous();
}
bool prepare_valid(OptTensor& v, int64_t batch, const Tensor& like) {
    if (!v || !v->defined()) { v.reset(); return true; }
    if (!v->has_storage() || v->layout() != at::kStrided || v->key_set().has(c10::DispatchKey::Python) || v->numel() != batch || v->is_floating_point() || v->is_complex() ||
        v->requires_grad())
        return false;
    v = v->to(like.device(), at::kInt).reshape({batch}).contiguous();
    return true;
}

// ---------------------------------------------------------------- the operator on (N, T, C) tensors
struct Cfg {
    int64_t N, T, C, heads, win, left, dil;
    double scale, drop_p;
    uint64_t seed;
};

void op_forward(const Tensor& o, const Tensor& lse, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& r, const Tensor& vl, const Cfg& c) {
    if (c.drop_p != 0.0)
        check(na1d_fused_forward_dropout(ptr(o), fptr(lse), ptr(q), ptr(k), ptr(v), fptr(r), static_cast<int32_t*>(ptr(vl)), c.N, c.heads, c.T, c.C,
                                         c.win, c.left, c.dil, (float)c.scale, (float)c.drop_p, c.seed, code(q), stream()),
              "na1d_fused_forward_dropout");
    else
        check(na1d_fused_forward(ptr(o), fptr(lse), ptr(q), ptr(k), ptr(v), fptr(r), static_cast<int32_t*>(ptr(vl)), c.N, c.heads, c.T, c.C, c.win,
                                 c.left, c.dil, (float)c.scale, code(q), stream()),
              "na1d_fused_forward");
}

struct NA1dFused : public torch::autograd::Function<NA1dFused> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& rpb, const OptTensor& vl,
                          int64_t heads, int64_t win, int64_t left, int64_t dil, double scale, double drop_p, int64_t seed) {
        const Cfg c{q.size(0), q.size(1), q.size(2), heads, win, left, dil, scale, drop_p, (uint64_t)seed};
        Tensor o = at::empty_like(q), lse = empty_f32({c.N, c.T}, q);
        const Tensor valid = vl ? *vl : Tensor();
        op_forward(o, lse, q, k, v, rpb32(rpb), valid, c);
        ctx->save_for_backward({q, k, v, o, lse, rpb ? *rpb : Tensor(), valid});
        auto& d = ctx->saved_data;
        d["heads"] = heads; d["win"] = win; d["left"] = left; d["dil"] = dil; d["scale"] = scale; d["drop_p"] = drop_p; d["seed"] = seed;
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        const Tensor &q = s[0], &k = s[1], &v = s[2], &o = s[3], &lse = s[4], &rpb = s[5], &vl = s[6];
        auto& d = ctx->saved_data;
        const Cfg c{q.size(0), q.size(1), q.size(2), d["heads"].toInt(), d["win"].toInt(), d["left"].toInt(), d["dil"].toInt(), d["scale"].toDouble(),
                    d["drop_p"].toDouble(), (uint64_t)d["seed"].toInt()};
        const c10::cuda::CUDAGuard guard(q.device());
        const Tensor d_o = grads[0].defined() ? grads[0].contiguous() : at::zeros_like(q);
        Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v), d_rpb;
        if (rpb.defined() && ctx->needs_input_grad(3)) d_rpb = zeros_f32(rpb.sizes(), q);
        // (a workspace that is not needed is not touched)
        const int64_t floats = c.drop_p != 0.0 ? c.N * c.T
                                               : na1d_fused_backward_workspace_floats(c.N, c.heads, c.T, c.C, c.win, c.left, c.dil, code(q), rpb.defined(), d_rpb.defined());
        const Tensor delta = floats == 0 ? lse : empty_f32({c.N, c.T}, q);
        const Tensor r = rpb32(rpb);
        if (c.drop_p != 0.0)
            check(na1d_fused_backward_dropout(ptr(dq), ptr(dk), ptr(dv), fptr(d_rpb), ptr(d_o), ptr(q), ptr(k), ptr(v), fptr(lse), fptr(r),
                                              static_cast<int32_t*>(ptr(vl)), fptr(delta), c.N * c.T, c.N, c.heads, c.T, c.C, c.win, c.left, c.dil,
                                              (float)c.scale, (float)c.drop_p, c.seed, code(q), stream()),
                  "na1d_fused_backward_dropout");
        else
            check(na1d_fused_backward(ptr(dq), ptr(dk), ptr(dv), fptr(d_rpb), ptr(d_o), ptr(q), ptr(k), ptr(v), ptr(o), fptr(lse), fptr(r),
                                      static_cast<int32_t*>(ptr(vl)), fptr(delta), c.N, c.heads, c.T, c.C, c.win, c.left, c.dil, (float)c.scale, code(q),
                                      stream()),
                  "na1d_fused_backward");
        if (d_rpb.defined()) d_rpb = d_rpb.to(rpb.scalar_type());
        return {dq, dk, dv, d_rpb, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

OptTensor fused(const Tensor& q, const Tensor& k, const Tensor& v, int64_t win, int64_t left, int64_t dil, double scale, OptTensor rpb, OptTensor vl,
                int64_t heads, double drop_p, uint64_t seed) {
    if (!eager_mode() || !plain16(q) || !plain16(k) || !plain16(v) || q.dim() != 3 || q.sizes() != k.sizes() || q.sizes() != v.sizes() ||
        q.scalar_type() != k.scalar_type() || q.scalar_type() != v.scalar_type() || q.device() != k.device() || q.device() != v.device() ||
        !q.is_contiguous() || !k.is_contiguous() || !v.is_contiguous() || heads <= 0 || win <= 0 || q.size(0) % heads != 0 || q.numel() == 0 ||
        !prepare_rpb(rpb, heads * win, q))
        return std::nullopt;
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    if (!prepare_valid(vl, q.size(0) / heads, q)) return std::nullopt;
    if (rpb && !rpb->defined()) rpb.reset();
    if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad() || (rpb && rpb->requires_grad())))
        return NA1dFused::apply(q, k, v, rpb, vl, heads, win, left, dil, scale, drop_p, (int64_t)seed);
    const Cfg c{q.size(0), q.size(1), q.size(2), heads, win, left, dil, scale, drop_p, seed};
    Tensor o = at::empty_like(q);
    op_forward(o, Tensor(), q, k, v, rpb32(rpb), vl ? *vl : Tensor(), c);
    return o;
}

// ---------------------------------------------------------------- the drop-in pair: q.k^T over the window, and its product with v
// rows (N, T, C) 16-bit, band (N, T, win) fp32; the six entry points differ in which of the three they write
struct Band {
    int64_t N, T, C, win, left, dil;
    Band(const Tensor& rows, int64_t win_, int64_t left_, int64_t dil_)
        : N(rows.size(0)), T(rows.size(1)), C(rows.size(2)), win(win_), left(left_), dil(dil_) {}
    Tensor products(int (*f)(float*, const void*, const void*, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int, void*), const char* name,
                    const Tensor& a, const Tensor& b) const {
        Tensor out = empty_f32({N, T, win}, a);
        check(f(fptr(out), ptr(a), ptr(b), N, T, C, win, left, dil, code(a), stream()), name);
        return out;
    }
    Tensor rows(int (*f)(void*, const float*, const void*, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int, void*), const char* name,
                const Tensor& band, const Tensor& x) const {
        Tensor out = at::empty_like(x);
        check(f(ptr(out), fptr(band), ptr(x), N, T, C, win, left, dil, code(x), stream()), name);
        return out;
    }
};
void keep_window(AutogradContext* ctx, int64_t win, int64_t left, int64_t dil) {
    auto& d = ctx->saved_data;
    d["win"] = win; d["left"] = left; d["dil"] = dil;
}
Band kept_window(AutogradContext* ctx, const Tensor& rows) {
    auto& d = ctx->saved_data;
    return Band(rows, d["win"].toInt(), d["left"].toInt(), d["dil"].toInt());
}

struct NA1dQK : public torch::autograd::Function<NA1dQK> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, int64_t win, int64_t left, int64_t dil) {
        ctx->save_for_backward({q, k});
        keep_window(ctx, win, left, dil);
        return Band(q, win, left, dil).products(na1d_qk_forward, "na1d_qk_forward", q, k);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        const Band b = kept_window(ctx, s[0]);
        const c10::cuda::CUDAGuard guard(s[0].device());
        const Tensor g = grads[0].defined() ? grads[0].contiguous() : at::zeros({b.N, b.T, b.win}, s[0].options().dtype(at::kFloat));
        Tensor dq = b.rows(na1d_q_backward, "na1d_q_backward", g, s[1]);
        return {dq, b.rows(na1d_k_backward, "na1d_k_backward", g, s[0]), Tensor(), Tensor(), Tensor()};
    }
};
struct NA1dAV : public torch::autograd::Function<NA1dAV> {
    static Tensor forward(AutogradContext* ctx, const Tensor& attn, const Tensor& v, int64_t win, int64_t left, int64_t dil) {
        ctx->save_for_backward({attn, v});
        keep_window(ctx, win, left, dil);
        return Band(v, win, left, dil).rows(na1d_av_forward, "na1d_av_forward", attn, v);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        const Band b = kept_window(ctx, s[1]);
        const c10::cuda::CUDAGuard guard(s[1].device());
        const Tensor g = grads[0].defined() ? grads[0].contiguous() : at::zeros_like(s[1]);
        Tensor da = b.products(na1d_a_backward, "na1d_a_backward", g, s[1]);
        return {da, b.rows(na1d_v_backward, "na1d_v_backward", s[0], g), Tensor(), Tensor(), Tensor()};
    }
};

bool band_rows(const Tensor& t) { return plain16(t) && t.dim() == 3 && t.numel() != 0 && t.is_contiguous(); }
OptTensor qk(const Tensor& q, const Tensor& k, int64_t win, int64_t left, int64_t dil, bool bf16) {
    if (!eager_mode() || !band_rows(q) || !band_rows(k) || q.sizes() != k.sizes() || q.device() != k.device() || win <= 0 ||
        q.scalar_type() != k.scalar_type() || q.scalar_type() != (bf16 ? at::kBFloat16 : at::kHalf))
        return std::nullopt;
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad())) return NA1dQK::apply(q, k, win, left, dil);
    return Band(q, win, left, dil).products(na1d_qk_forward, "na1d_qk_forward", q, k);
}
OptTensor av(const Tensor& attn, const Tensor& v, int64_t win, int64_t left, int64_t dil, bool bf16) {
    if (!eager_mode() || !band_rows(v) || !plain(attn) || attn.scalar_type() != at::kFloat || !attn.is_contiguous() || attn.dim() != 3 ||
        attn.size(0) != v.size(0) || attn.size(1) != v.size(1) || attn.size(2) != win || attn.device() != v.device() ||
        v.scalar_type() != (bf16 ? at::kBFloat16 : at::kHalf))
        return std::nullopt;
    const c10::cuda::OptionalCUDAGuard guard(v.device());
    if (at::GradMode::is_enabled() && (attn.requires_grad() || v.requires_grad())) return NA1dAV::apply(attn, v, win, left, dil);
    return Band(v, win, left, dil).rows(na1d_av_forward, "na1d_av_forward", attn, v);
}

// ---------------------------------------------------------------- the operator on a packed (batch, T, 3, heads, C) tensor
struct Packed {
    int64_t B, T, H, C, win, left, dil;
    double scale;
    int64_t in[3], out[3];   // {batch, head, token} element strides of q, k, v and of o
    Packed(int64_t B_, int64_t T_, int64_t D, int64_t heads, int64_t win_, int64_t left_, int64_t dil_, double scale_)
        : B(B_), T(T_), H(heads), C(D / heads), win(win_), left(left_), dil(dil_), scale(scale_), in{T * 3 * D, C, 3 * D}, out{T * D, C, D} {}
    Packed(const Tensor& qkv, int64_t heads, int64_t win_, int64_t left_, int64_t dil_, double scale_)
        : Packed(qkv.size(0), qkv.size(1), qkv.size(2) / 3, heads, win_, left_, dil_, scale_) {}
};
void packed_forward(const Tensor& o, const Tensor& lse, const Tensor& qkv, const Tensor& r, const Tensor& vl, const Packed& c) {
    char* p = static_cast<char*>(ptr(qkv));
    const int64_t step = c.H * c.C * 2;
    check(na1d_fused_forward_strided(ptr(o), fptr(lse), p, p + step, p + 2 * step, fptr(r), static_cast<int32_t*>(ptr(vl)), c.out, c.in, c.in, c.in,
                                     c.B * c.H, c.H, c.T, c.C, c.win, c.left, c.dil, (float)c.scale, code(qkv), stream()),
          "na1d_fused_forward_strided");
}
void packed_backward(const Tensor& d_qkv, const Tensor& d_rpb, const Tensor& d_o, const Tensor& qkv, const Tensor& lse, const Tensor& r, const Tensor& vl,
                     const Packed& c) {
    char *p = static_cast<char*>(ptr(qkv)), *g = static_cast<char*>(ptr(d_qkv));
    const int64_t step = c.H * c.C * 2, n = d_rpb.defined() ? 160 * c.H * c.win : 0;   // one partial row per CTA (one CTA per SM)
    Tensor scratch;
    if (n) scratch = empty_f32({n}, qkv);
    check(na1d_fused_backward_strided(g, g + step, g + 2 * step, fptr(d_rpb), ptr(d_o), p, p + step, p + 2 * step, fptr(lse), fptr(r),
                                      static_cast<int32_t*>(ptr(vl)), fptr(scratch), n, c.in, c.in, c.in, c.out, c.in, c.in, c.in, c.B * c.H, c.H, c.T,
                                      c.C, c.win, c.left, c.dil, (float)c.scale, code(qkv), stream()),
          "na1d_fused_backward_strided");
}

struct NA1dFusedPacked : public torch::autograd::Function<NA1dFusedPacked> {
    static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const OptTensor& rpb, const OptTensor& vl, int64_t heads, int64_t win, int64_t left,
                          int64_t dil, double scale) {
        const Packed c(qkv, heads, win, left, dil, scale);
        Tensor o = at::empty({c.B, c.T, c.H * c.C}, qkv.options()), lse = empty_f32({c.B * c.H, c.T}, qkv);
        const Tensor valid = vl ? *vl : Tensor();
        packed_forward(o, lse, qkv, rpb32(rpb), valid, c);
        ctx->save_for_backward({qkv, lse, rpb ? *rpb : Tensor(), valid});
        auto& d = ctx->saved_data;
        d["heads"] = heads; d["win"] = win; d["left"] = left; d["dil"] = dil; d["scale"] = scale;
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        const Tensor &qkv = s[0], &lse = s[1], &rpb = s[2], &vl = s[3];
        auto& d = ctx->saved_data;
        const Packed c(qkv, d["heads"].toInt(), d["win"].toInt(), d["left"].toInt(), d["dil"].toInt(), d["scale"].toDouble());
        const c10::cuda::CUDAGuard guard(qkv.device());
        const Tensor d_o = grads[0].defined() ? grads[0].contiguous() : at::zeros({c.B, c.T, c.H * c.C}, qkv.options());
        Tensor d_qkv = at::empty_like(qkv), d_rpb;
        if (rpb.defined() && ctx->needs_input_grad(1)) d_rpb = zeros_f32(rpb.sizes(), qkv);
        packed_backward(d_qkv, d_rpb, d_o, qkv, lse, rpb32(rpb), vl, c);
        if (d_rpb.defined()) d_rpb = d_rpb.to(rpb.scalar_type());
        return {d_qkv, d_rpb, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

OptTensor packed(const Tensor& qkv, int64_t heads, int64_t win, int64_t left, int64_t dil, double scale, OptTensor rpb, OptTensor vl) {
    if (!eager_mode() || !plain16(qkv) || qkv.dim() != 3 || qkv.numel() == 0 || !qkv.is_contiguous() || heads <= 0 || win <= 0 ||
        qkv.size(2) % (3 * heads) != 0 || !prepare_rpb(rpb, heads * win, qkv))
        return std::nullopt;
    const c10::cuda::OptionalCUDAGuard guard(qkv.device());
    if (!prepare_valid(vl, qkv.size(0), qkv)) return std::nullopt;
    if (rpb && !rpb->defined()) rpb.reset();
    if (at::GradMode::is_enabled() && (qkv.requires_grad() || (rpb && rpb->requires_grad())))
        return NA1dFusedPacked::apply(qkv, rpb, vl, heads, win, left, dil, scale);
    const Packed c(qkv, heads, win, left, dil, scale);
    Tensor o = at::empty({c.B, c.T, c.H * c.C}, qkv.options());
    packed_forward(o, Tensor(), qkv, rpb32(rpb), vl ? *vl : Tensor(), c);
    return o;
}

// An output gradient as the row and column kernels read it: dense, on a 16-byte boundary (a view into another tensor need not be).
Tensor aligned(const Tensor& g, uintptr_t bytes = 16) {
    const Tensor c = g.contiguous();
    return (reinterpret_cast<uintptr_t>(c.data_ptr()) & (bytes - 1)) ? c.clone() : c;
}

// What a node of more than the operator saved, as the kernels read it, wherever a saved-tensor hook has put it.
variable_list saved_dense(AutogradContext* ctx) {
    variable_list saved = ctx->get_saved_variables();
    const at::NoGradGuard off;
    for (Tensor& t : saved)
        if (t.defined() && t.is_cuda()) t = aligned(t);
    return saved;
}

// A backward pass works in the types of its forward, also where it is called under autocast (to another type, the library products
// would hand the kernels tensors of that type).
struct NoAutocast {
    const c10::impl::ExcludeDispatchKeyGuard guard{c10::autocast_dispatch_keyset};
};

// ---------------------------------------------------------------- backward passes that are differentiated again
// Under create_graph a backward has to be differentiable itself, and the kernels' results are not. There a node with more in it than
// the attention takes its branch again in PyTorch's operations (the attention as the operator's own node, whose gradients are
// constants to a second pass) and differentiates that. The inputs come from what the node saved, and stand in the graph where the
// node's own inputs do; each behind an alias, at which the inner pass ends.
Tensor stand_in(const Tensor& data, size_t edge) {
    const torch::autograd::Edge& e = torch::autograd::get_current_node()->next_edge(edge);
    const Tensor t = data.detach();
    if (!e.is_valid()) return t;
    torch::autograd::impl::set_gradient_edge(t, e);
    return at::alias(t);
}
// gradients of `outputs` with respect to the stand-ins, undefined for those whose input wants none
variable_list inner_gradients(const variable_list& outputs, const variable_list& inputs, const variable_list& grads) {
    variable_list out, in, g;
    for (size_t i = 0; i < outputs.size(); ++i)
        if (grads[i].defined()) { out.push_back(outputs[i]); g.push_back(grads[i]); }
    for (const Tensor& t : inputs)
        if (t.defined() && t.requires_grad()) in.push_back(t);
    variable_list result(inputs.size());
    if (out.empty() || in.empty()) return result;
    const variable_list found = torch::autograd::grad(out, in, g, true, true, true);
    for (size_t i = 0, k = 0; i < inputs.size(); ++i)
        if (inputs[i].defined() && inputs[i].requires_grad()) result[i] = found[k++];
    return result;
}

// Shapes that the strided entry points do not take (a head size outside theirs, no shared memory left for the bias gradient): the
// heads are split and merged by one copy each around the dense ones.
bool takes_packed(const Packed& c, const Tensor& like, bool backward = true) {
    return na1d_fused_strided_supported(c.H, c.T, c.C, c.win, c.left, c.dil, code(like), 1, backward) == 1;
}
Tensor heads_moved(const Tensor& in, const Packed& c, int64_t parts, bool to_dense) {
    Tensor out = to_dense ? at::empty({parts, c.B * c.H, c.T, c.C}, in.options()) : at::empty({c.B, c.T, parts * c.H * c.C}, in.options());
    check(na1d_permute_heads(ptr(out), ptr(in), c.B, c.T, parts, c.H, c.C, to_dense, stream()), "na1d_permute_heads");
    return out;
}
Cfg dense_cfg(const Packed& c) { return Cfg{c.B * c.H, c.T, c.C, c.H, c.win, c.left, c.dil, c.scale, 0.0, 0}; }
// the attention on a packed qkv by either route; o_dense, and the split qkv in the place of the packed one: what the dense route's backward reads
void attention_forward(Tensor& o, Tensor& o_dense, Tensor& qkv, const Tensor& lse, const Tensor& r, const Tensor& vl, const Packed& c, bool packed) {
    if (packed) {
        o = at::empty({c.B, c.T, c.H * c.C}, qkv.options());
        packed_forward(o, lse, qkv, r, vl, c);
        return;
    }
    qkv = heads_moved(qkv, c, 3, true);
    o_dense = at::empty({c.B * c.H, c.T, c.C}, qkv.options());
    op_forward(o_dense, lse, qkv.select(0, 0), qkv.select(0, 1), qkv.select(0, 2), r, vl, dense_cfg(c));
    o = heads_moved(o_dense, c, 1, false);
}
// gradient of the packed qkv; d_o (rows, D)
Tensor attention_backward(const Tensor& d_rpb, const Tensor& d_o, const Tensor& qkv, const Tensor& o_dense, const Tensor& lse, const Tensor& r, const Tensor& vl,
                          const Packed& c) {
    Tensor d_qkv = at::empty_like(qkv);
    if (!o_dense.defined()) {
        packed_backward(d_qkv, d_rpb, d_o, qkv, lse, r, vl, c);
        return d_qkv;
    }
    const Tensor moved = heads_moved(d_o, c, 1, true), delta = empty_f32({c.B * c.H, c.T}, qkv);
    auto part = [](const Tensor& t, int i) { return ptr(t.select(0, i)); };
    check(na1d_fused_backward(part(d_qkv, 0), part(d_qkv, 1), part(d_qkv, 2), fptr(d_rpb), ptr(moved), part(qkv, 0), part(qkv, 1), part(qkv, 2), ptr(o_dense), fptr(lse),
                              fptr(r), static_cast<int32_t*>(ptr(vl)), fptr(delta), c.B * c.H, c.H, c.T, c.C, c.win, c.left, c.dil, (float)c.scale, code(qkv),
                              stream()),
          "na1d_fused_backward");
    return heads_moved(d_qkv, c, 3, false);
}

// ---------------------------------------------------------------- the transformer block
// Whether the weight-gradient kernel takes these products (M, N: their sizes). It has a pair of SMs to a tile of 256 x 256 and splits the rows
// where that leaves pairs idle; with few splits or none a sum over partial tiles is left of its gain, which the library's products do not
// pay, and only many rows make up for it. In us, kernel / library with column sums: more than two splits (an MLP of 256 channels, 8 tiles)
// 2400 rows 18 / 23, 38400 rows 48 / 88; two (a layer of 768, an MLP of 512; 36 and 32 tiles) 600 rows 27 / 19 and 24 / 18, 2400 rows
// 31 / 30 and 30 / 30, 9600 rows 51 / 61 and 49 / 61; none (an MLP of 640, a layer of 1024; 60 and 64 tiles) 2400 rows 43 / 34 and
// 46 / 36, 9600 rows 83 / 75 and 87 / 85, 38400 rows 261 / 281 and 276 / 294; more tiles than pairs (an MLP of 1024, 128 tiles) 2400 rows
// 83 / 50, 38400 rows 538 / 506.
bool gradients_in_one_launch(const int64_t* M, const int64_t* N, int n, int64_t rows) {
    const int64_t pairs = std::max(1, at::cuda::getCurrentDeviceProperties()->multiProcessorCount / 2);
    int64_t tiles = 0;
    for (int i = 0; i < n; ++i) tiles += ((M[i] + 255) / 256) * ((N[i] + 255) / 256);
    return tiles * (rows < 4800 ? 3 : rows < 20000 ? 2 : 1) <= pairs;
}
// Parameter gradients of up to two projections: d_w = dy^T x and d_b = column sums of dy, of `type` from fp32 sums.
// dy (rows, M), x (rows, N); what is not wanted stays undefined.
struct ParameterGrads {
    Tensor w[2], b[2];
    ParameterGrads(const Tensor (&dy)[2], const Tensor (&x)[2], const bool (&need_w)[2], const bool (&need_b)[2], at::ScalarType type) {
        void *pw[2], *pb[2];
        const void *py[2], *px[2];
        int64_t M[2], N[2];
        int n = 0;
        const int64_t rows = dy[0].size(0);
        for (int i = 0; i < 2; ++i) {
            if (!need_w[i]) continue;
            M[n] = dy[i].size(1);
            N[n] = x[i].size(1);
            ++n;
        }
        const bool one = n > 0 && gradients_in_one_launch(M, N, n, rows);
        n = 0;
        for (int i = 0; i < 2; ++i) {
            if (one && need_w[i]) {
                const auto opts = dy[i].options().dtype(type);
                w[i] = at::empty({M[n], N[n]}, opts);
                if (need_b[i]) b[i] = at::empty({M[n]}, opts);
                pw[n] = ptr(w[i]); pb[n] = ptr(b[i]); py[n] = ptr(dy[i]); px[n] = ptr(x[i]);
                ++n;
                continue;
            }
            if (need_w[i]) w[i] = at::mm(dy[i].t(), x[i], at::kFloat).to(type);
            if (need_b[i]) b[i] = column_sums(dy[i]).to(type);
        }
        if (!one) return;
        const Tensor scratch = empty_f32({na1d_projection_gradients_scratch(M, N, n, rows)}, dy[0]);
        check(na1d_projection_gradients(pw, pb, py, px, M, N, n, rows, fptr(scratch), type == at::kFloat, code(dy[0]), stream()), "na1d_projection_gradients");
    }
    static Tensor column_sums(const Tensor& dy) {
        const int64_t rows = dy.size(0), F = dy.size(1);
        const Tensor sums = empty_f32({F}, dy), scratch = empty_f32({na1d_block_scratch_floats(rows, 0, F)}, dy);
        check(na1d_column_sums(fptr(sums), fptr(scratch), ptr(dy), rows, F, code(dy), stream()), "na1d_column_sums");
        return sums;
    }
};

// Parameters in the order qkv.w, qkv.b, proj.w, proj.b, fc1.w, fc1.b, fc2.w, fc2.b, norm1.w, norm1.b, norm2.w, norm2.b, bias table.
constexpr int kProj = 8, kParams = 13;
constexpr int64_t kSlot = 64;   // elements: 128-byte slots of the packed 16-bit parameters

struct Projections {
    Tensor buf, t[kProj];
    void views(at::IntArrayRef (&shapes)[kProj]) {
        int64_t off = buf.storage_offset();   // (what a saved-tensor hook gives back may lie inside another tensor)
        for (int i = 0; i < kProj; ++i) {
            const int64_t n = c10::multiply_integers(shapes[i]);
            t[i] = shapes[i].size() == 2 ? buf.as_strided(shapes[i], {shapes[i][1], 1}, off) : buf.as_strided(shapes[i], {1}, off);
            off += (n + kSlot - 1) / kSlot * kSlot;
        }
    }
    void cast(const Tensor* params, const Tensor& like) {
        const float* src[kProj];
        int64_t dst[kProj], n[kProj], total = 0;
        at::IntArrayRef shapes[kProj];
        for (int i = 0; i < kProj; ++i) {
            shapes[i] = params[i].sizes();
            src[i] = fptr(params[i]);
            n[i] = params[i].numel();
            dst[i] = total;
            total += (n[i] + kSlot - 1) / kSlot * kSlot;
        }
        buf = at::empty({total}, like.options());
        check(na1d_cast_parameters(ptr(buf), src, dst, n, kProj, code(like), stream()), "na1d_cast_parameters");
        views(shapes);
    }
};

struct BlockState {   // what the backward needs
    Tensor s1, st1, h1, qkv, lse, o, s2, st2, h2, f, g, buf, o_dense;
};
// one row of padding keeps both halves of the statistics 16-byte aligned
inline Tensor row_stats(int64_t rows, const Tensor& like) { return empty_f32({2, (rows + 3) / 4 * 4}, like); }

void layer_norm(Tensor& y, Tensor& sum, Tensor& st, const Tensor& x, const Tensor& dx, const Tensor& w, const Tensor& b, double eps, bool stats) {
    const int64_t D = x.size(2), rows = x.size(0) * x.size(1);
    y = at::empty_like(x);
    sum = dx.defined() ? at::empty_like(x) : x;
    if (stats) st = row_stats(rows, x);
    check(na1d_layer_norm_forward(ptr(y), dx.defined() ? ptr(sum) : nullptr, fptr(st), stats ? fptr(st) + st.size(1) : nullptr, ptr(x), ptr(dx), fptr(w),
                                  fptr(b), rows, D, (float)eps, code(x), stream()),
          "na1d_layer_norm_forward");
}
// its column sums stay in parts, in `part`
Tensor layer_norm_backward(const Tensor& dy, const Tensor& s, const Tensor& st, const Tensor& w, const Tensor& res, float* part) {
    const int64_t D = s.size(2);
    Tensor ds = at::empty_like(s);
    check(na1d_layer_norm_backward_rows(ptr(ds), part, ptr(dy), ptr(s), fptr(st), fptr(st) + st.size(1), fptr(w), ptr(res), s.size(0) * s.size(1), D, code(s),
                                        stream()),
          "na1d_layer_norm_backward_rows");
    return ds;
}

// Whether a block's evaluation takes its MLP as one kernel. A tile of 256 rows is a chain of pieces on a pair of SMs (sums over the hidden
// layer are not split there, so that both routes give the same bits): 7 us and 2.3 us for a piece of 128 columns in every round of
// pairs, against 9 us and 0.063 us for a tile's piece in the passes. Hidden size 1024, passes / kernel in us: 2400 rows 15 / 26, 9600 rows
// 28 / 27, 38400 rows 81 / 64, 153600 rows 314 / 175.
bool mlp_pays(int64_t rows, int64_t F) {
    const int64_t tiles = (rows + 255) / 256, pairs = std::max(1, at::cuda::getCurrentDeviceProperties()->multiProcessorCount / 2);
    const double pieces = F / 128.0;
    return 7 + 2.3 * pieces * ((tiles + pairs - 1) / pairs) <= 9 + 0.063 * pieces * tiles;
}

// x (+ dx): the residual stream. Returns the stream after the attention branch and the MLP branch's output; their sum is the
// block's output, taken inside the next block's first LayerNorm. Where the MLP kernel runs, the sum alone (the second tensor
// undefined), without a backward pass to come in `out` if that is given: rows of D inside wider ones.
std::pair<Tensor, Tensor> block_forward(const Tensor& x, const Tensor& dx, const Tensor& vl, const Packed& c, double eps1, double eps2,
                                        const Tensor* p, BlockState* keep, const OptTensor& out = std::nullopt) {
    const int64_t D = x.size(2), rows = c.B * c.T;
    const bool stats = keep != nullptr;
    BlockState st;
    Projections w;
    w.cast(p, x);
    layer_norm(st.h1, st.s1, st.st1, x, dx, p[8], p[9], eps1, stats);
    st.qkv = product(st.h1.view({rows, D}), w.t[0], w.t[1], false).view({c.B, c.T, 3 * D});
    if (stats) st.lse = empty_f32({c.B * c.H, c.T}, x);
    attention_forward(st.o, st.o_dense, st.qkv, st.lse, p[12], vl, c, takes_packed(c, x, stats));
    const Tensor y = product(st.o.view({rows, D}), w.t[2], w.t[3], false).view({c.B, c.T, D});
    layer_norm(st.h2, st.s2, st.st2, st.s1, y, p[10], p[11], eps2, stats);
    const int64_t F = w.t[4].size(0), floats = na1d_mlp_scratch_floats(rows, D, F);
    Tensor s2, z;
    if (floats >= 0 && (keep || mlp_pays(rows, F))) {
        const Tensor scratch = floats && keep ? empty_f32({floats}, x) : Tensor();
        s2 = out && !keep ? *out : at::empty_like(x);
        if (keep) st.f = at::empty({rows, F}, x.options());
        check(na1d_mlp_forward_rounded(ptr(s2), s2.stride(1), ptr(st.f), ptr(st.s2), ptr(st.h2), ptr(w.t[4]), ptr(w.t[5]), ptr(w.t[6]), ptr(w.t[7]), fptr(scratch),
                                       rows, D, F, code(x), stream()),
              "na1d_mlp_forward_rounded");
    } else {
        st.f = product(st.h2.view({rows, D}), w.t[4], w.t[5], false);
        st.g = at::empty_like(st.f);
        check(na1d_gelu_forward(ptr(st.g), ptr(st.f), st.f.numel(), code(x), stream()), "na1d_gelu_forward");
        z = product(st.g, w.t[6], w.t[7], false).view({c.B, c.T, D});
        s2 = st.s2;
    }
    if (keep) {
        st.buf = w.buf;
        *keep = std::move(st);
    }
    return {s2, z};
}

// ---------------------------------------------------------------- a projection of tensors side by side
// y = cat(parts) w^T + b, and the parts themselves for what reads them next: their gradients then come through this node, which adds its own
// share inside the product that makes it. (Summed by autograd instead, the 20 contributions of a network of six stages were slices
// of wider gradients, 27 us each at 38400 rows of 256 where the products with the addition take 11 to 13; the bias gradient, a column sum
// of 54 us, comes with the weight gradient.)
struct NA1dFuse : public torch::autograd::Function<NA1dFuse> {
    static variable_list forward(AutogradContext* ctx, const Tensor& weight, const Tensor& bias, at::TensorList parts) {
        const Tensor& x = parts[0];
        const int64_t D = x.size(2), rows = x.size(0) * x.size(1), O = weight.size(0), K = weight.size(1);
        const float* src[2] = {fptr(weight), fptr(bias)};
        const int64_t n[2] = {O * K, O}, dst[2] = {0, (O * K + kSlot - 1) / kSlot * kSlot};
        const Tensor buf = at::empty({dst[1] + O}, x.options());
        check(na1d_cast_parameters(ptr(buf), src, dst, n, 2, code(x), stream()), "na1d_cast_parameters");
        const Tensor w = buf.as_strided({O, K}, {K, 1}, 0), b = buf.as_strided({O}, {1}, dst[1]);
        const Tensor cat = parts.size() == 1 ? x : at::cat(parts, 2);
        const Tensor y = product(cat.view({rows, K}), w, b, false).view({x.size(0), x.size(1), O});
        ctx->save_for_backward({cat, buf});
        ctx->saved_data["D"] = D;
        ctx->saved_data["O"] = O;
        ctx->set_materialize_grads(false);
        variable_list out = {y};
        out.insert(out.end(), parts.begin(), parts.end());
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = saved_dense(ctx);
        const Tensor &cat = s[0], &buf = s[1];
        const int64_t D = ctx->saved_data["D"].toInt(), O = ctx->saved_data["O"].toInt(), K = cat.size(2), rows = cat.size(0) * cat.size(1), parts = K / D;
        const c10::cuda::CUDAGuard guard(cat.device());
        const NoAutocast off;
        const Tensor w = buf.narrow(0, 0, O * K).view({O, K}), b = buf.narrow(0, (O * K + kSlot - 1) / kSlot * kSlot, O);
        if (at::GradMode::is_enabled()) {
            variable_list in = {stand_in(w.to(at::kFloat), 0), stand_in(b.to(at::kFloat), 1)}, out = {Tensor()};
            for (int64_t i = 0; i < parts; ++i) in.push_back(stand_in(cat.narrow(2, i * D, D), 2 + i));
            out.insert(out.end(), in.begin() + 2, in.end());
            out[0] = at::linear(at::cat(variable_list(in.begin() + 2, in.end()), 2), in[0].to(w.scalar_type()), in[1].to(w.scalar_type()));
            for (size_t i = 0; i < out.size(); ++i)
                if (!out[i].requires_grad()) grads[i] = Tensor();
            return inner_gradients(out, in, grads);
        }
        variable_list result(2 + parts);
        const Tensor dy = grads[0].defined() ? aligned(grads[0]).view({rows, O}) : Tensor();
        for (int64_t i = 0; i < parts; ++i) {
            if (!ctx->needs_input_grad(2 + i)) continue;
            const Tensor& more = grads[1 + i];
            if (!dy.defined()) {
                result[2 + i] = more;
                continue;
            }
            // rows of a wider gradient are read in place
            Tensor add;
            if (more.defined()) {
                const bool in_place = more.stride(2) == 1 && more.stride(1) % 8 == 0 && more.stride(1) >= D && more.stride(0) == more.stride(1) * more.size(1) &&
                                      more.storage_offset() >= 0 && (reinterpret_cast<uintptr_t>(more.data_ptr()) & 15u) == 0;
                add = in_place ? more.as_strided({rows, D}, {more.stride(1), 1}) : aligned(more).view({rows, D});
            }
            result[2 + i] = product(dy, w.narrow(1, i * D, D), Tensor(), true, add).view({cat.size(0), cat.size(1), D});
        }
        if (dy.defined()) {
            const Tensor x = cat.view({rows, K});
            const ParameterGrads g({dy, dy}, {x, x}, {ctx->needs_input_grad(0), false}, {ctx->needs_input_grad(1), false}, at::kFloat);
            result[0] = g.w[0];
            result[1] = g.b[0];
        }
        return result;
    }
};

std::vector<Tensor> fuse(const Tensor& weight, const Tensor& bias, const std::vector<Tensor>& parts) {
    TORCH_CHECK(!parts.empty() && weight.size(1) == (int64_t)parts.size() * parts[0].size(2), "a fused projection takes parts of one width");
    const c10::cuda::OptionalCUDAGuard guard(parts[0].device());
    return NA1dFuse::apply(weight, bias, at::TensorList(parts));
}

struct NA1dBlock : public torch::autograd::Function<NA1dBlock> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& dx, const OptTensor& vl, int64_t heads, int64_t win, int64_t left,
                                 double scale, double eps1, double eps2, const Tensor& p0, const Tensor& p1, const Tensor& p2, const Tensor& p3,
                                 const Tensor& p4, const Tensor& p5, const Tensor& p6, const Tensor& p7, const Tensor& p8, const Tensor& p9,
                                 const Tensor& p10, const Tensor& p11, const Tensor& p12) {
        const Tensor p[kParams] = {p0, p1, p2, p3, p4, p5, p6, p7, p8, p9, p10, p11, p12};
        const Packed c(x.size(0), x.size(1), x.size(2), heads, win, left, 1, scale);
        BlockState st;
        auto out = block_forward(x, dx ? *dx : Tensor(), vl ? *vl : Tensor(), c, eps1, eps2, p, &st);
        ctx->save_for_backward({st.s1, st.st1, st.h1, st.qkv, st.lse, st.o, st.s2, st.st2, st.h2, st.f, st.g, st.buf, p8, p10, p12, vl ? *vl : Tensor(), p9, p11, st.o_dense});
        auto& d = ctx->saved_data;
        d["heads"] = heads; d["win"] = win; d["left"] = left; d["scale"] = scale; d["dx"] = dx.has_value(); d["eps1"] = eps1; d["eps2"] = eps2;
        return out.second.defined() ? variable_list{out.first, out.second} : variable_list{out.first};
    }
    // x, dx, then the parameters; w: the 16-bit ones
    static variable_list differentiable(const variable_list& s, const Packed& c, const Projections& w, double eps1, double eps2, bool has_dx, int first,
                                        const variable_list& grads) {
        const Tensor &s1 = s[0], &vl = s[15];
        const int64_t D = s1.size(2);
        const auto half = s1.scalar_type();
        variable_list in = {stand_in(s1, 0), has_dx ? stand_in(at::zeros_like(s1), 1) : Tensor()};
        for (int i = 0; i < kProj; ++i) in.push_back(stand_in(w.t[i].to(at::kFloat), first + i));
        const int norms[5] = {12, 16, 13, 17, 14};   // n1w, n1b, n2w, n2b, bias table among the saved tensors
        for (int i = 0; i < 5; ++i) in.push_back(stand_in(s[norms[i]], first + kProj + i));
        const Tensor* p = &in[2];
        auto linear = [&](const Tensor& x, int i) { return at::linear(x, p[i].to(half), p[i + 1].to(half)); };
        auto norm = [&](const Tensor& x, int i, double eps) { return at::layer_norm(x.to(at::kFloat), {D}, p[i], p[i + 1], eps).to(half); };
        const Tensor x = has_dx ? in[0] + in[1] : in[0];
        const OptTensor valid = vl.defined() ? OptTensor(vl) : OptTensor();
        const Tensor qkv = linear(norm(x, 8, eps1), 0);
        Tensor o;
        if (!s[18].defined()) {
            o = NA1dFusedPacked::apply(qkv, p[12], valid, c.H, c.win, c.left, 1, c.scale);
        } else {
            const Tensor q = qkv.view({c.B, c.T, 3, c.H, c.C}).permute({2, 0, 3, 1, 4}).contiguous().view({3, c.B * c.H, c.T, c.C});
            o = NA1dFused::apply(q.select(0, 0), q.select(0, 1), q.select(0, 2), OptTensor(p[12]), valid, c.H, c.win, c.left, 1, c.scale, 0.0, (int64_t)0)
                    .view({c.B, c.H, c.T, c.C}).transpose(1, 2).reshape({c.B, c.T, D});
        }
        const Tensor s2 = x + linear(o, 2);
        const Tensor z = linear(at::gelu(linear(norm(s2, 10, eps2), 4)), 6);
        return inner_gradients(grads.size() == 1 ? variable_list{s2 + z} : variable_list{s2, z}, in, grads);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = saved_dense(ctx);
        const Tensor &s1 = s[0], &st1 = s[1], &h1 = s[2], &qkv = s[3], &lse = s[4], &o = s[5], &s2 = s[6], &st2 = s[7], &h2 = s[8], &buf = s[11], &n1w = s[12],
                     &n2w = s[13], &rpb = s[14], &vl = s[15];
        const Tensor f = aligned(s[9], 32);   // (read by whole sectors)
        Tensor g = s[10];
        auto& data = ctx->saved_data;
        const Packed c(s1.size(0), s1.size(1), s1.size(2), data["heads"].toInt(), data["win"].toInt(), data["left"].toInt(), 1, data["scale"].toDouble());
        const c10::cuda::CUDAGuard guard(s1.device());
        const NoAutocast off;
        const bool has_dx = data["dx"].toBool();
        const int first = 1 + (has_dx ? 1 : 0) + (vl.defined() ? 1 : 0);   // edge of the first parameter
        auto need = [&](int k) { return ctx->needs_input_grad(first + k); };
        const int64_t D = s1.size(2), rows = c.B * c.T, F = f.size(1);
        const std::vector<int64_t> shapes[kProj] = {{3 * D, D}, {3 * D}, {D, D}, {D}, {F, D}, {F}, {D, F}, {D}};
        at::IntArrayRef refs[kProj];
        for (int i = 0; i < kProj; ++i) refs[i] = shapes[i];
        Projections w;
        w.buf = buf;
        w.views(refs);
        if (at::GradMode::is_enabled()) {
            const variable_list g = differentiable(s, c, w, data["eps1"].toDouble(), data["eps2"].toDouble(), has_dx, first, grads);
            const Tensor none;
            variable_list out = {g[0], g[1], none, none, none, none, none, none, none};
            out.insert(out.end(), g.begin() + 2, g.end());
            return out;
        }
        // partial column sums of GELU's and the two norms' passes, one after the other
        const int64_t room = (na1d_block_scratch_floats(rows, D, std::max(F, 3 * D)) + 3) / 4 * 4;
        const Tensor scratch = empty_f32({2 * room}, s1);
        const bool one = grads.size() == 1;   // the output is s2 + z, from the MLP kernel
        const Tensor d_s2 = grads[0].defined() ? aligned(grads[0]) : one ? at::zeros_like(s2) : Tensor();
        const Tensor d_z = (one ? d_s2 : grads[1].defined() ? aligned(grads[1]) : at::zeros_like(s2)).view({rows, D});
        // MLP branch
        Tensor d_b1, d_f = at::empty_like(f), d_h;
        if (one) {
            const int64_t floats = na1d_mlp_scratch_floats(rows, D, F);
            const Tensor part = floats ? empty_f32({floats}, s1) : Tensor();
            d_h = at::empty_like(s2);
            g = at::empty_like(f);
            check(na1d_mlp_backward(ptr(d_h), ptr(d_f), ptr(g), ptr(d_z), ptr(f), ptr(w.t[4]), ptr(w.t[6]), fptr(part), rows, D, F, code(f), stream()),
                  "na1d_mlp_backward");
        } else {
            const Tensor d_g = product(d_z, w.t[6], Tensor(), true);
            d_b1 = empty_f32({F}, s1);
            check(na1d_gelu_backward(ptr(d_f), fptr(d_b1), fptr(scratch), ptr(d_g), ptr(f), rows, F, code(f), stream()), "na1d_gelu_backward");
            d_h = product(d_f, w.t[4], Tensor(), true);
        }
        const ParameterGrads mlp({d_f, d_z}, {h2.view({rows, D}), g}, {need(4), need(6)}, {one && need(5), need(7)}, at::kFloat);
        if (one) d_b1 = mlp.b[0];
        d_f.reset();
        g.reset();
        const Tensor sums = empty_f32({2, 3, D}, s1), sums1 = sums.select(0, 0), sums2 = sums.select(0, 1);
        const Tensor d_y = layer_norm_backward(d_h, s2, st2, n2w, d_s2, fptr(scratch) + room);   // also the residual stream's gradient
        // attention branch
        const Tensor dy2 = d_y.view({rows, D});
        Tensor d_rpb;
        if (need(12)) d_rpb = zeros_f32(rpb.sizes(), s1);
        const Tensor d_qkv = attention_backward(d_rpb, product(dy2, w.t[2], Tensor(), true), qkv, s[18], lse, rpb, vl, c);
        const Tensor dq2 = d_qkv.view({rows, 3 * D});
        const ParameterGrads att({dq2, dy2}, {h1.view({rows, D}), o.view({rows, D})}, {need(0), need(2)}, {need(1), false}, at::kFloat);
        const Tensor d_x = layer_norm_backward(product(dq2, w.t[0], Tensor(), true), s1, st1, n1w, d_y, fptr(scratch));
        check(na1d_layer_norm_sums(fptr(sums1), fptr(sums2), fptr(scratch), fptr(scratch) + room, rows, D, stream()), "na1d_layer_norm_sums");
        const Tensor none;
        return {d_x, has_dx ? d_x : none, none, none, none, none, none, none, none, att.w[0], att.b[0], att.w[1], sums2.select(0, 2), mlp.w[0], d_b1, mlp.w[1],
                mlp.b[1],
                sums1.select(0, 0), sums1.select(0, 1), sums2.select(0, 0), sums2.select(0, 1), d_rpb};
    }
};

// out: 16-byte aligned slices of wider rows for the result, without gradients (a hint: what comes back is the result).
// nothing where the valid lengths are not of a form the kernels can be given (on another device, or of another integer type, they are
// converted)
std::optional<std::pair<Tensor, Tensor>> block(const Tensor& x, const OptTensor& dx, OptTensor vl, int64_t heads, int64_t win, int64_t left, double scale,
                                               double eps1, double eps2, const std::vector<Tensor>& p, const OptTensor& out) {
    TORCH_CHECK(p.size() == kParams, "a block has 13 parameters");
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    if (!prepare_valid(vl, x.size(0), x)) return std::nullopt;
    if (at::GradMode::is_enabled()) {
        const variable_list r = NA1dBlock::apply(x, dx, vl, heads, win, left, scale, eps1, eps2, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8],
                                                 p[9], p[10], p[11], p[12]);
        return std::make_pair(r[0], r.size() > 1 ? r[1] : Tensor());
    }
    const Packed c(x.size(0), x.size(1), x.size(2), heads, win, left, 1, scale);
    return block_forward(x, dx ? *dx : Tensor(), vl ? *vl : Tensor(), c, eps1, eps2, p.data(), nullptr, out);
}

// ---------------------------------------------------------------- the attention layer
// Channels first ((N, C, T) in and out, grouped 1x1 convolutions): the layout changes once on the C-channel input and once on
// the output; in between both convolutions are one GEMM each over all N*T tokens (dense block-diagonal weights: at these
// sizes the tensor cores make the zeros free), their rows ordered so that the result is the packed tensor the attention reads.
// Channels last ((N, T, C), linear projections): the projections as they are. In both, parameters are rounded to 16 bits by one
// launch per projection (or layer) and bias gradients are column sums of this library.
struct LayerShape {
    int64_t B, T, D, groups;
    bool first;
    LayerShape(const Tensor& x, bool first_, int64_t groups_)
        : B(x.size(0)), T(x.size(first_ ? 2 : 1)), D(x.size(first_ ? 1 : 2)), groups(groups_), first(first_) {}
    int64_t rows() const { return B * T; }
};
struct LayerWeights {
    Tensor qw, qb, pw, pb;   // 16-bit, dense (3D, D), (3D), (D, D), (D); biases may be undefined
    LayerWeights(const Tensor& x, const LayerShape& l, const Tensor& qw_, const OptTensor& qb_, const Tensor& pw_, const OptTensor& pb_) {
        const Tensor src[4] = {qw_, qb_ ? *qb_ : Tensor(), pw_, pb_ ? *pb_ : Tensor()};
        Tensor* dst[4] = {&qw, &qb, &pw, &pb};
        const int64_t n[4] = {3 * l.D * l.D, 3 * l.D, l.D * l.D, l.D};
        const bool src32 = qw_.scalar_type() == at::kFloat;
        if (l.first || src32) {
            const Tensor buf = at::empty({n[0] + n[1] + n[2] + n[3] + 4 * kSlot}, x.options());
            const float* from[4];
            int64_t offs[4], sizes[4], off = 0;
            int count = 0;
            for (int i = 0; i < 4; ++i) {
                if (!src[i].defined()) continue;
                *dst[i] = i & 1 ? buf.as_strided({n[i]}, {1}, off) : buf.as_strided({n[i] / l.D, l.D}, {l.D, 1}, off);
                from[count] = fptr(src[i]); offs[count] = off; sizes[count] = n[i]; ++count;
                off += (n[i] + kSlot - 1) / kSlot * kSlot;
            }
            if (l.first) {
                check(na1d_pack_grouped(ptr(qw), ptr(qb), ptr(src[0]), ptr(src[1]), src32, l.D, l.groups, 3, code(x), stream()), "na1d_pack_grouped");
                check(na1d_pack_grouped(ptr(pw), ptr(pb), ptr(src[2]), ptr(src[3]), src32, l.D, l.groups, 1, code(x), stream()), "na1d_pack_grouped");
            } else {
                check(na1d_cast_parameters(ptr(buf), from, offs, sizes, count, code(x), stream()), "na1d_cast_parameters");
            }
        } else {
            for (int i = 0; i < 4; ++i) *dst[i] = src[i].defined() ? src[i].detach() : Tensor();
        }
    }
};
Tensor project(const Tensor& x, const Tensor& w, const Tensor& b) { return product(x, w, b, false); }
Tensor transposed(const Tensor& in, const LayerShape& l, bool to_tokens) {
    Tensor out = to_tokens ? at::empty({l.B, l.T, l.D}, in.options()) : at::empty({l.B, l.D, l.T}, in.options());
    check(na1d_transpose(ptr(out), ptr(in), l.B, l.D, l.T, to_tokens, code(in), stream()), "na1d_transpose");
    return out;
}
// gradients of the two projections' parameters, fp32 sums in the parameters' own type, shape and order: 0 = qkv, 1 = proj
struct LayerGrads {
    Tensor w[2], b[2];
    LayerGrads(const bool (&need_w)[2], const bool (&need_b)[2], const Tensor (&dy)[2], const Tensor (&x)[2], const at::IntArrayRef (&w_shape)[2],
               at::ScalarType type, const LayerShape& l) {
        const ParameterGrads dense(dy, x, need_w, need_b, l.first ? at::kFloat : type);
        for (int i = 0; i < 2; ++i) {
            const int parts = i == 0 ? 3 : 1;
            w[i] = dense.w[i];
            b[i] = dense.b[i];
            if (!l.first || (!need_w[i] && !need_b[i])) continue;
            const auto opts = dy[i].options().dtype(type);
            if (need_w[i]) w[i] = at::empty(w_shape[i], opts);
            if (need_b[i]) b[i] = at::empty({parts * l.D}, opts);
            check(na1d_unpack_grouped(ptr(w[i]), ptr(b[i]), fptr(dense.w[i]), fptr(dense.b[i]), type == at::kFloat, l.D, l.groups, parts, code(dy[i]), stream()),
                  "na1d_unpack_grouped");
        }
    }
};
// qkv: packed, or (dense) the split one; o_dense: the dense route's own output
struct LayerState { Tensor xt, qkv, lse, o, qw, pw, o_dense, qb, pb; };
Tensor layer_forward(const Tensor& x, const LayerShape& l, const Tensor& vl, const Tensor& r, const Tensor& qw, const OptTensor& qb, const Tensor& pw,
                     const OptTensor& pb, const Packed& c, LayerState* keep) {
    const LayerWeights w(x, l, qw, qb, pw, pb);
    LayerState s;
    s.xt = l.first ? transposed(x, l, true) : x;
    s.qkv = project(s.xt.view({l.rows(), l.D}), w.qw, w.qb).view({l.B, l.T, 3 * l.D});
    if (keep) s.lse = empty_f32({l.B * c.H, l.T}, x);
    attention_forward(s.o, s.o_dense, s.qkv, s.lse, r, vl, c, takes_packed(c, x));
    Tensor y = project(s.o.view({l.rows(), l.D}), w.pw, w.pb);
    y = l.first ? transposed(y, l, false) : y.view({l.B, l.T, l.D});
    if (keep) { s.qw = w.qw; s.pw = w.pw; s.qb = w.qb; s.pb = w.pb; *keep = std::move(s); }
    return y;
}
struct NA1dLayer : public torch::autograd::Function<NA1dLayer> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& rpb, const Tensor& qw, const Tensor& pw, const OptTensor& qb,
                          const OptTensor& pb, const OptTensor& vl, bool first, int64_t heads, int64_t groups, int64_t win, int64_t left, int64_t dil,
                          double scale) {
        const LayerShape l(x, first, groups);
        const Packed c(l.B, l.T, l.D, heads, win, left, dil, scale);
        LayerState s;
        Tensor y = layer_forward(x, l, vl ? *vl : Tensor(), rpb32(rpb), qw, qb, pw, pb, c, &s);
        ctx->save_for_backward({s.xt, s.qkv, s.lse, s.o, s.qw, s.pw, rpb, vl ? *vl : Tensor(), s.o_dense, s.qb, s.pb});
        auto& d = ctx->saved_data;
        d["first"] = first; d["heads"] = heads; d["groups"] = groups; d["win"] = win; d["left"] = left; d["dil"] = dil; d["scale"] = scale;
        d["qb"] = qb.has_value(); d["pb"] = pb.has_value();
        d["qw_shape"] = qw.sizes().vec(); d["pw_shape"] = pw.sizes().vec(); d["type"] = (int64_t)qw.scalar_type();
        return y;
    }
    // a projection's weight and bias in their own type, shape and order, from the 16-bit dense ones
    static std::pair<Tensor, Tensor> parameters(const Tensor& w, const Tensor& b, at::IntArrayRef shape, at::ScalarType type, const LayerShape& l, int parts) {
        if (!l.first) return {w.to(type), b.defined() ? b.to(type) : Tensor()};
        const Tensor out_w = at::empty(shape, w.options().dtype(type)), out_b = b.defined() ? at::empty({parts * l.D}, w.options().dtype(type)) : Tensor();
        const Tensor dense = w.to(at::kFloat), sums = b.defined() ? b.to(at::kFloat) : Tensor();
        check(na1d_unpack_grouped(ptr(out_w), ptr(out_b), fptr(dense), fptr(sums), type == at::kFloat, l.D, l.groups, parts, code(w), stream()),
              "na1d_unpack_grouped");
        return {out_w, out_b};
    }
    // x, rpb, qkv weight, projection weight, qkv bias, projection bias
    static variable_list differentiable(const variable_list& s, const LayerShape& l, const Packed& c, at::IntArrayRef qw_shape, at::IntArrayRef pw_shape,
                                        at::ScalarType type, const Tensor& dy) {
        const Tensor &xt = s[0], &rpb = s[6], &vl = s[7], &qb = s[9], &pb = s[10];
        const auto half = xt.scalar_type();
        const auto q = parameters(s[4], qb, qw_shape, type, l, 3), p = parameters(s[5], pb, pw_shape, type, l, 1);
        const variable_list in = {stand_in(l.first ? transposed(xt, l, false) : xt, 0), stand_in(rpb, 1), stand_in(q.first, 2), stand_in(p.first, 3),
                                  qb.defined() ? stand_in(q.second, 4) : Tensor(), pb.defined() ? stand_in(p.second, qb.defined() ? 5 : 4) : Tensor()};
        auto project_with = [&](const Tensor& x, int i) {
            const OptTensor b = in[i + 2].defined() ? OptTensor(in[i + 2].to(half)) : OptTensor();
            return l.first ? at::conv1d(x, in[i].to(half), b, 1, at::IntArrayRef({0}), 1, l.groups) : at::linear(x, in[i].to(half), b.value_or(Tensor()));
        };
        Tensor y = project_with(in[0], 2);
        // head split and merge (models/PCF_NATransformer.py:126-138, 151)
        y = l.first ? y.view({l.B, l.D / l.groups, l.groups, 3, l.T}).transpose(1, 2).reshape({l.B, c.H, c.C, 3, l.T}).permute({3, 0, 1, 4, 2})
                    : y.view({l.B, l.T, 3, c.H, c.C}).permute({2, 0, 3, 1, 4});
        y = y.contiguous().view({3, l.B * c.H, l.T, c.C});
        y = NA1dFused::apply(y.select(0, 0), y.select(0, 1), y.select(0, 2), OptTensor(in[1]), vl.defined() ? OptTensor(vl) : OptTensor(), c.H, c.win, c.left,
                             c.dil, c.scale, 0.0, (int64_t)0)
                .view({l.B, c.H, l.T, c.C});
        y = l.first ? y.transpose(2, 3).reshape({l.B, l.D, l.T}) : y.transpose(1, 2).reshape({l.B, l.T, l.D});
        return inner_gradients({project_with(y, 3)}, in, {dy});
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = saved_dense(ctx);
        const Tensor &xt = s[0], &qkv = s[1], &lse = s[2], &o = s[3], &qw = s[4], &pw = s[5], &rpb = s[6], &vl = s[7], &o_dense = s[8];
        auto& d = ctx->saved_data;
        const Packed c(xt.size(0), xt.size(1), xt.size(2), d["heads"].toInt(), d["win"].toInt(), d["left"].toInt(), d["dil"].toInt(), d["scale"].toDouble());
        LayerShape l(xt, false, d["groups"].toInt());
        l.first = d["first"].toBool();
        const c10::cuda::CUDAGuard guard(qkv.device());
        const NoAutocast off;
        const auto type = (at::ScalarType)d["type"].toInt();
        const bool has_qb = d["qb"].toBool(), has_pb = d["pb"].toBool();
        const int qb_edge = 4, pb_edge = 4 + (has_qb ? 1 : 0);
        if (at::GradMode::is_enabled()) {
            variable_list out = differentiable(s, l, c, d["qw_shape"].toIntVector(), d["pw_shape"].toIntVector(), type, grads[0]);
            out.resize(14);
            return out;
        }
        Tensor dy = grads[0].defined() ? aligned(grads[0]) : at::zeros(l.first ? at::IntArrayRef({l.B, l.D, l.T}) : xt.sizes(), xt.options());
        dy = (l.first ? transposed(dy, l, true) : dy).view({l.rows(), l.D});
        Tensor d_rpb, d_x;
        if (ctx->needs_input_grad(1)) d_rpb = zeros_f32(rpb.sizes(), xt);
        const Tensor d_qkv = attention_backward(d_rpb, product(dy, pw, Tensor(), true), qkv, o_dense, lse, rpb32(rpb), vl, c);
        const Tensor dq = d_qkv.view({l.rows(), 3 * l.D});
        const std::vector<int64_t> qw_shape = d["qw_shape"].toIntVector(), pw_shape = d["pw_shape"].toIntVector();
        const LayerGrads g({ctx->needs_input_grad(2), ctx->needs_input_grad(3)},
                           {has_qb && ctx->needs_input_grad(qb_edge), has_pb && ctx->needs_input_grad(pb_edge)}, {dq, dy},
                           {xt.view({l.rows(), l.D}), o.view({l.rows(), l.D})}, {qw_shape, pw_shape}, type, l);
        if (ctx->needs_input_grad(0)) {
            d_x = product(dq, qw, Tensor(), true);
            d_x = l.first ? transposed(d_x, l, false) : d_x.view({l.B, l.T, l.D});
        }
        if (d_rpb.defined()) d_rpb = d_rpb.to(rpb.scalar_type());
        const Tensor none;
        return {d_x, d_rpb, g.w[0], g.w[1], g.b[0], g.b[1], none, none, none, none, none, none, none, none};
    }
};

// sizes that every kernel of the node takes, in either direction (the operator itself refuses the same sizes on every route)
bool layer_fits(const LayerShape& l, int64_t heads, bool cast) {
    const int64_t rows = l.rows(), C = l.D / heads;
    return l.D <= (l.first ? 8192 : (1 << 20) / 3) && (!cast || l.first || 3 * l.D * l.D <= INT32_MAX / 16) && (!l.first || l.T <= 1 << 20) &&
           rows <= INT32_MAX / 2 && rows <= (1ll << 40) / (3 * l.D) && l.T <= INT32_MAX / 8 && l.T * C <= (int64_t)INT32_MAX * 4 && C <= 4096;
}
// 16-bit x; weights and biases all of x's type, or (under autocast to x's type) all fp32
OptTensor layer(const Tensor& x, bool first, const OptTensor& bias, const Tensor& qw, const OptTensor& qb, const Tensor& pw, const OptTensor& pb,
                int64_t heads, int64_t groups, int64_t win, int64_t left, int64_t dil, double scale, OptTensor vl) {
    if (!bias || !bias->defined()) return std::nullopt;   // (a layer without a bias table: its modules)
    const Tensor& rpb = *bias;
    if (!eager_mode() || !plain16(x) || x.dim() != 3 || x.numel() == 0 || !x.is_contiguous() || x.size(0) > 65535 || heads <= 0 || win <= 0 || groups <= 0)
        return std::nullopt;
    const LayerShape l(x, first, groups);
    const bool cast = at::autocast::is_autocast_enabled(at::kCUDA);
    const auto type = qw.scalar_type();
    if ((cast && at::autocast::get_autocast_dtype(at::kCUDA) != x.scalar_type()) || (type != x.scalar_type() && !(cast && type == at::kFloat)) || l.D % 8 != 0 ||
        l.D % groups != 0 || l.D % heads != 0 || (!first && groups != 1) || !layer_fits(l, heads, type == at::kFloat) || !prepare_rpb(rpb, heads * win, x))
        return std::nullopt;
    auto fits = [&](const Tensor& t, int64_t n) { return plain(t) && t.device() == x.device() && t.scalar_type() == type && t.is_contiguous() && t.numel() == n; };
    if (!fits(qw, 3 * l.D * (l.D / groups)) || !fits(pw, l.D * (l.D / groups)) || (qb && !fits(*qb, 3 * l.D)) || (pb && !fits(*pb, l.D))) return std::nullopt;
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    if (!prepare_valid(vl, l.B, x)) return std::nullopt;
    if (at::GradMode::is_enabled() && (x.requires_grad() || rpb.requires_grad() || qw.requires_grad() || pw.requires_grad() ||
                                       (qb && qb->requires_grad()) || (pb && pb->requires_grad())))
        return NA1dLayer::apply(x, rpb, qw, pw, qb, pb, vl, first, heads, groups, win, left, dil, scale);
    return layer_forward(x, l, vl ? *vl : Tensor(), rpb32(rpb), qw, qb, pw, pb, Packed(l.B, l.T, l.D, heads, win, left, dil, scale), nullptr);
}

// int32 (N): clamp(T - padding, 0, T); padding of one element counts for every utterance
OptTensor valid_tokens(const Tensor& padding, int64_t T, int64_t N) {
    if (!eager_mode() || !plain(padding) || (padding.scalar_type() != at::kInt && padding.scalar_type() != at::kLong) || !padding.is_contiguous() ||
        padding.dim() > 1 || (padding.numel() != 1 && padding.numel() != N) || N <= 0 || T <= 0 || T > INT32_MAX)
        return std::nullopt;
    const c10::cuda::OptionalCUDAGuard guard(padding.device());
    Tensor out = at::empty({N}, padding.options().dtype(at::kInt));
    check(na1d_valid_tokens(static_cast<int32_t*>(ptr(out)), ptr(padding), padding.scalar_type() == at::kLong, padding.numel(), N, T, stream()),
          "na1d_valid_tokens");
    return out;
}

}  // namespace

PYBIND11_MODULE(_na1d_torch, m) {
    // without the interpreter lock, as PyTorch's own operators: a launch may wait for room in the stream's queue
#define NA1D_DEF(f) m.def(#f, torch::wrap_pybind_function_no_gil(f))
    NA1D_DEF(fused);
    NA1D_DEF(qk);
    NA1D_DEF(av);
    NA1D_DEF(packed);
    NA1D_DEF(block);
    NA1D_DEF(fuse);
    NA1D_DEF(layer);
    NA1D_DEF(valid_tokens);
#undef NA1D_DEF
    m.def("eager_mode", &eager_mode);
}
