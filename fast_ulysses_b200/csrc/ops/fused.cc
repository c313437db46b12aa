#include "fused.hpp"

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <nvtx3/nvToolsExt.h>
#include <torch/autograd.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>

namespace py = pybind11;

namespace fu {
namespace {

using at::Tensor;
using MaybeTensor = std::optional<at::Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int64_t kHeadDim = 128;

struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&)            = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};

void ok(int rc)
{
    TORCH_CHECK(rc == FU_OK, "fast_ulysses_b200 kernel launch refused (", rc, "): ", fu_last_error());
}

// An argument check of a Python entry point: AssertionError, as its `assert` would raise.
template <class... Args>
void expect(bool good, const Args&... what)
{
    if (!good) {
        const std::string              text = c10::str(what...);
        const py::gil_scoped_acquire   gil;
        PyErr_SetString(PyExc_AssertionError, text.c_str());
        throw py::error_already_set();
    }
}

// Operands of one launch lie on one GPU: an address of another device, or of the host, would reach the
// kernels as if it were this one's.
void expect_on_device_of(const Tensor& x, std::initializer_list<const Tensor*> operands, const char* what)
{
    expect(x.is_cuda(), what, ": expected CUDA tensors, got one on ", x.device());
    for (const Tensor* t : operands) {
        if (t->defined()) {
            expect(t->device() == x.device(), what, ": expected every operand on ", x.device(), ", got one on ", t->device());
        }
    }
}

// What an epilogue reads beside a product of `rows` x w.size(0): one bias value per column, and a residual with
// the product's values, which it reads as bf16.
void expect_epilogue(const Tensor& w, const Tensor& bias, const Tensor& residual, int64_t rows, const char* what)
{
    const int64_t n = w.size(0);
    if (bias.defined()) {
        expect(bias.numel() == n, what, ": expected a bias of ", n, " values, got ", bias.sizes());
    }
    if (residual.defined()) {
        expect(residual.scalar_type() == at::kBFloat16 && residual.numel() == rows * n, what, ": expected a bf16 residual of ", rows,
               " rows of ", n, " values, got ", residual.scalar_type(), " ", residual.sizes());
    }
}

cudaStream_t stream_of(const Tensor& t)
{
    return at::cuda::getCurrentCUDAStream(t.device().index());
}

// One device word per GPU that kernels set when one of their bounded waits ran out.
Tensor error_word(int64_t device)
{
    const c10::Device          dev(c10::DeviceType::CUDA, static_cast<c10::DeviceIndex>(device));
    const c10::cuda::CUDAGuard on(dev);
    void*                      word = nullptr;
    ok(fu_error_word(&word));
    return at::from_blob(word, {1}, at::TensorOptions().dtype(at::kInt).device(dev));
}

uint32_t* error_ptr(const Tensor& t)
{
    // asked for once per device and thread
    static thread_local uint32_t* cached[16] = {};
    const int64_t                 d = t.device().index();
    if (d < 0 || d >= 16) {
        return static_cast<uint32_t*>(error_word(d).data_ptr());
    }
    if (!cached[d]) {
        cached[d] = static_cast<uint32_t*>(error_word(d).data_ptr());
    }
    return cached[d];
}

// A tensor that starts on 16 bytes, as vector loads need, with its strides: a gradient can be a view of any offset.
Tensor aligned(const Tensor& t)
{
    return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone();
}

Tensor empty_bf16(at::IntArrayRef shape, const Tensor& like)
{
    return at::detail::empty_cuda(shape, at::kBFloat16, like.device(), std::nullopt);
}
// `t` with the strides of `out`, which an epilogue reads it by: a tensor saved for backward comes back dense where
// hooks have packed it (moved to the host, say), whatever its pitch was.
Tensor laid_out_like(const Tensor& out, const Tensor& t)
{
    if (t.strides() == out.strides() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0) {
        return t;
    }
    Tensor copy = at::empty_strided(out.sizes(), out.strides(), out.options());
    copy.copy_(t);
    return copy;
}

// A matrix of this library's own, read by later GEMMs: rows on 32-byte sectors, which TMA moves up to 1.7 times
// as fast as rows that are not.
Tensor empty_operand(int64_t rows, int64_t cols, const Tensor& like)
{
    return cols % 16 == 8 ? empty_bf16({rows, cols + 8}, like).narrow(1, 0, cols) : empty_bf16({rows, cols}, like);
}
Tensor empty_f32(at::IntArrayRef shape, const Tensor& like)
{
    return at::detail::empty_cuda(shape, at::kFloat, like.device(), std::nullopt);
}

// Whether a call goes through its autograd node. A forward-mode tangent does too, whatever the grad mode: the node
// has no rule for one and says so, instead of a result without it.
bool wants_grad(std::initializer_list<const Tensor*> ts)
{
    const bool reverse = at::GradMode::is_enabled();
    for (const Tensor* t : ts) {
        if (t->defined() && ((reverse && t->requires_grad()) || t->_fw_grad(/*level=*/0).defined())) {
            return true;
        }
    }
    return false;
}

Tensor or_none(const MaybeTensor& t)
{
    return t.has_value() ? *t : Tensor();
}
MaybeTensor maybe(const Tensor& t)
{
    return t.defined() ? MaybeTensor(t) : std::nullopt;
}

// Which gradients of a node are wanted, by argument. Autograd numbers a node's inputs without the
// optional tensors that were not given.
class Wanted {
public:
    Wanted(AutogradContext* ctx, std::initializer_list<bool> given)
    {
        size_t edge = 0;
        for (const bool g : given) {
            wanted_.push_back(g && ctx->needs_input_grad(edge));
            edge += g ? 1 : 0;
        }
    }
    bool operator[](size_t i) const { return wanted_[i]; }

private:
    std::vector<bool> wanted_;
};

// ---- GEMM -----------------------------------------------------------------------------------------------
// A view whose rows are contiguous and start 16 bytes apart (copying if needed).
Tensor tma_ready(const Tensor& x)
{
    if (x.stride(1) == 1 && x.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0) {
        return x;
    }
    const int64_t rows = x.size(0), cols = x.size(1);
    Tensor        buf  = at::empty({rows, (cols + 7) / 8 * 8}, x.options());
    Tensor        out  = buf.narrow(1, 0, cols);
    out.copy_(x);
    return out;
}

struct GemmExtra {
    Tensor  bias, residual, aux, store_pre, out;
    int     act  = 0;
    bool    a_km = false, b_kn = false;
    int64_t ctas = 0;
    int     flags = 0;
};

Tensor gemm(const Tensor& a_in, const Tensor& b_in, const GemmExtra& x = {})
{
    const Tensor  a = tma_ready(a_in), b = tma_ready(b_in);
    const int64_t k = a.size(x.a_km ? 0 : 1), m = a.size(x.a_km ? 1 : 0);
    const int64_t n = b.size(x.b_kn ? 1 : 0);
    Tensor        out = x.out.defined() ? x.out : empty_bf16({m, n}, a);
    FuGemmArgs    g{};
    g.a   = a.data_ptr();
    g.b   = b.data_ptr();
    g.c   = out.data_ptr();
    g.m   = m;
    g.n   = n;
    g.k   = k;
    g.lda = a.stride(0);
    g.ldb = b.stride(0);
    g.ldc = out.stride(0);
    g.flags = x.flags | (x.a_km ? FU_GEMM_A_KM : 0) | (x.b_kn ? FU_GEMM_B_KN : 0);
    if (x.bias.defined()) {
        g.bias = x.bias.data_ptr();
        if (x.bias.scalar_type() == at::kBFloat16) {
            g.flags |= FU_GEMM_BIAS_BF16;
        }
    }
    g.residual = x.residual.defined() ? x.residual.data_ptr() : nullptr;
    g.aux      = x.aux.defined() ? x.aux.data_ptr() : nullptr;
    g.c_pre    = x.store_pre.defined() ? x.store_pre.data_ptr() : nullptr;
    g.act      = x.act;
    g.ctas     = static_cast<int32_t>(x.ctas);
    g.err      = error_ptr(a);
    ok(fu_gemm_bf16(&g, stream_of(a)));
    return out;
}

Tensor gemm_entry(const Tensor& a, const Tensor& b, const MaybeTensor& bias, const MaybeTensor& residual, int64_t act,
                  const MaybeTensor& out, int64_t ctas, bool a_km, bool b_kn, const MaybeTensor& aux,
                  const MaybeTensor& store_pre, std::optional<bool> pair)
{
    expect(a.is_cuda() && b.is_cuda() && a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16,
           "gemm_bf16: a and b must be bf16 CUDA tensors");
    expect(a.dim() == 2 && b.dim() == 2, "gemm_bf16: a and b must be matrices");
    const int64_t m = a.size(a_km ? 1 : 0), n = b.size(b_kn ? 1 : 0);
    expect(a.size(a_km ? 0 : 1) == b.size(b_kn ? 0 : 1), "gemm_bf16: ", a.sizes(), " and ", b.sizes(),
           " do not share a contraction (a_km=", a_km, ", b_kn=", b_kn, ")");
    for (const MaybeTensor* t : {&bias, &residual, &out, &aux, &store_pre}) {
        const Tensor given = or_none(*t);
        expect_on_device_of(a, {&b, &given}, "gemm_bf16");
    }
    GemmExtra x;
    x.act  = static_cast<int>(act);
    x.a_km = a_km;
    x.b_kn = b_kn;
    x.ctas = ctas;
    x.flags = pair.has_value() ? (*pair ? FU_GEMM_PAIR : FU_GEMM_SINGLE) : 0;
    const c10::cuda::CUDAGuard on(a.device());
    x.out = out.has_value() ? *out : empty_bf16({m, n}, a);
    expect(x.out.dim() == 2 && x.out.size(0) == m && x.out.size(1) == n && x.out.stride(1) == 1
               && x.out.scalar_type() == at::kBFloat16,
           "gemm_bf16: out must be a bf16 (", m, ", ", n, ") matrix with dense rows");
    if (bias.has_value()) {
        expect(bias->scalar_type() == at::kFloat && bias->numel() == n && bias->is_contiguous(),
               "gemm_bf16: bias must be ", n, " dense fp32 values");
        x.bias = *bias;
    }
    if (residual.has_value()) {
        expect(residual->scalar_type() == at::kBFloat16 && residual->sizes() == x.out.sizes()
                   && residual->stride(0) == x.out.stride(0),
               "gemm_bf16: residual must be bf16 and laid out like the result");
        x.residual = *residual;
    }
    for (const MaybeTensor* t : {&aux, &store_pre}) {
        if (t->has_value()) {
            expect((*t)->scalar_type() == at::kBFloat16 && (*t)->sizes() == x.out.sizes() && (*t)->strides() == x.out.strides(),
                   "gemm_bf16: aux and store_pre must be bf16 and laid out like the result");
        }
    }
    x.aux       = or_none(aux);
    x.store_pre = or_none(store_pre);
    return gemm(a, b, x);
}

// Sum over the rows of a bf16 matrix, in fp32, rounded to the matrix' type: a bias gradient.
Tensor column_sum(const Tensor& g2)
{
    Tensor out = empty_bf16({g2.size(1)}, g2);
    ok(fu_colsum_bf16(g2.data_ptr(), out.data_ptr(), g2.size(0), g2.size(1), g2.stride(0), stream_of(g2)));
    return out;
}

// The bias as the epilogue can read it: bf16 or fp32 values without gaps.
Tensor bias_ready(const Tensor& bias)
{
    if (!bias.defined()) {
        return bias;
    }
    Tensor b = bias.scalar_type() == at::kBFloat16 || bias.scalar_type() == at::kFloat ? bias : bias.to(at::kFloat);
    return b.contiguous();
}

// A gradient in the type of what it is the gradient of.
Tensor as_type_of(const Tensor& g, const Tensor& grad_out)
{
    return g.scalar_type() == grad_out.scalar_type() ? g : g.to(grad_out.scalar_type());
}

Tensor rows_of(const Tensor& t, int64_t cols)
{
    return t.reshape({-1, cols});
}

std::vector<int64_t> shape_with_last(at::IntArrayRef shape, int64_t last)
{
    std::vector<int64_t> s = shape.vec();
    s.back()               = last;
    return s;
}

Tensor linear_forward(const Tensor& x2, const Tensor& w, const Tensor& bias, const Tensor& residual)
{
    GemmExtra e;
    e.bias = bias_ready(bias);
    if (residual.defined()) {
        e.residual = rows_of(residual, w.size(0)).contiguous();
    }
    return gemm(x2, w, e);
}

struct Linear : public torch::autograd::Function<Linear> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const MaybeTensor& bias,
                          const MaybeTensor& residual)
    {
        const at::AutoDispatchBelowAutograd below;
        const Tensor x2 = rows_of(x, x.size(-1));
        ctx->save_for_backward({x2, w});
        ctx->saved_data["x_shape"]  = x.sizes().vec();
        ctx->saved_data["bias"]     = bias.has_value();
        ctx->saved_data["residual"] = residual.has_value();
        return linear_forward(x2, w, or_none(bias), or_none(residual)).view(shape_with_last(x.sizes(), w.size(0)));
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        const at::AutoDispatchBelowADInplaceOrView below;
        const variable_list        saved = ctx->get_saved_variables();
        const Tensor               x2 = saved[0], w = saved[1], gy = grads[0];
        const c10::cuda::CUDAGuard on(gy.device());
        const Tensor               gy2 = rows_of(gy, gy.size(-1)).contiguous();
        const Wanted wanted(ctx, {true, true, ctx->saved_data["bias"].toBool(), ctx->saved_data["residual"].toBool()});
        variable_list              out(4);
        if (wanted[0]) {
            // dX[m, k] = sum_n dY[m, n] W[n, k]: W as stored is the (contraction x output) operand
            GemmExtra e;
            e.b_kn = true;
            out[0] = gemm(gy2, w, e).view(ctx->saved_data["x_shape"].toIntVector());
        }
        if (wanted[1]) {
            // dW[n, k] = sum_m dY[m, n] X[m, k]: both operands contract along their rows
            GemmExtra e;
            e.a_km = e.b_kn = true;
            out[1]          = gemm(gy2, x2, e);
        }
        if (wanted[2]) {
            out[2] = column_sum(gy2);
        }
        if (wanted[3]) {
            out[3] = gy;
        }
        return out;
    }
};

Tensor linear_entry(const Tensor& x, const Tensor& w, const MaybeTensor& bias, const MaybeTensor& residual)
{
    expect(x.is_cuda() && w.is_cuda() && x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16,
           "linear: x and weight must be bf16 CUDA tensors");
    expect(w.dim() == 2 && x.dim() >= 1 && x.size(-1) == w.size(1), "linear: ", x.sizes(), " x ", w.sizes());
    const Tensor b = or_none(bias), r = or_none(residual);
    expect_on_device_of(x, {&w, &b, &r}, "linear");
    expect_epilogue(w, b, r, c10::multiply_integers(x.sizes().slice(0, x.dim() - 1)), "linear");
    const c10::cuda::CUDAGuard on(x.device());
    if (wants_grad({&x, &w, &b, &r})) {
        return Linear::apply(x, w, maybe(b), maybe(r));
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    return linear_forward(rows_of(x, x.size(-1)), w, b, r).view(shape_with_last(x.sizes(), w.size(0)));
}

// gelu_tanh(x @ w1.T + b1) @ w2.T + b2 (+ residual): two GEMMs whose epilogues do everything else.
// Forward: GELU in the first one's epilogue, which also stores the pre-activation when a backward
// will want it; residual in the second's. Backward: the GELU's derivative is applied in the epilogue
// of the GEMM that produces its incoming gradient.
struct FeedForward : public torch::autograd::Function<FeedForward> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const MaybeTensor& b1, const Tensor& w2,
                          const MaybeTensor& b2, const MaybeTensor& residual)
    {
        const at::AutoDispatchBelowAutograd below;
        const Tensor x2 = rows_of(x, x.size(-1));
        GemmExtra    e;
        e.bias         = bias_ready(or_none(b1));
        e.act          = 1;
        e.store_pre    = empty_operand(x2.size(0), w1.size(0), x);
        e.out          = empty_operand(x2.size(0), w1.size(0), x);
        const Tensor h = gemm(x2, w1, e);
        ctx->save_for_backward({x2, w1, w2, e.store_pre, h});
        ctx->saved_data["x_shape"]  = x.sizes().vec();
        ctx->saved_data["b1"]       = b1.has_value();
        ctx->saved_data["b2"]       = b2.has_value();
        ctx->saved_data["residual"] = residual.has_value();
        return linear_forward(h, w2, or_none(b2), or_none(residual)).view(shape_with_last(x.sizes(), w2.size(0)));
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        const at::AutoDispatchBelowADInplaceOrView below;
        const variable_list        saved = ctx->get_saved_variables();
        const Tensor               x2 = saved[0], w1 = saved[1], w2 = saved[2], pre = saved[3], h = saved[4], gy = grads[0];
        const c10::cuda::CUDAGuard on(gy.device());
        const Tensor               gy2 = rows_of(gy, gy.size(-1)).contiguous();
        variable_list              out(6);
        const Wanted wanted(ctx, {true, true, ctx->saved_data["b1"].toBool(), true, ctx->saved_data["b2"].toBool(),
                                  ctx->saved_data["residual"].toBool()});
        GemmExtra                  wgrad;
        wgrad.a_km = wgrad.b_kn = true;
        if (wanted[3]) {
            out[3] = gemm(gy2, h, wgrad);
        }
        if (wanted[4]) {
            out[4] = column_sum(gy2);
        }
        if (wanted[0] || wanted[1] || wanted[2]) {
            GemmExtra e;  // d(pre-activation) = (gy W2) * gelu'(pre)
            e.b_kn = true;
            e.act  = 3;
            e.out  = empty_operand(gy2.size(0), w2.size(1), gy2);
            e.aux  = laid_out_like(e.out, pre);
            const Tensor gpre = gemm(gy2, w2, e);
            if (wanted[1]) {
                out[1] = gemm(gpre, x2, wgrad);
            }
            if (wanted[2]) {
                out[2] = column_sum(gpre);
            }
            if (wanted[0]) {
                GemmExtra d;
                d.b_kn = true;
                out[0] = gemm(gpre, w1, d).view(ctx->saved_data["x_shape"].toIntVector());
            }
        }
        if (wanted[5]) {
            out[5] = gy;
        }
        return out;
    }
};

Tensor feed_forward_entry(const Tensor& x, const Tensor& w1, const MaybeTensor& b1, const Tensor& w2, const MaybeTensor& b2,
                          const MaybeTensor& residual)
{
    expect(x.is_cuda() && x.scalar_type() == at::kBFloat16 && w1.scalar_type() == at::kBFloat16
               && w2.scalar_type() == at::kBFloat16,
           "feed_forward: x and both weights must be bf16 CUDA tensors");
    expect(w1.dim() == 2 && w2.dim() == 2 && x.dim() >= 1 && x.size(-1) == w1.size(1) && w2.size(1) == w1.size(0),
           "feed_forward: ", x.sizes(), " x ", w1.sizes(), " x ", w2.sizes());
    const Tensor  c1 = or_none(b1), c2 = or_none(b2), r = or_none(residual);
    const int64_t rows = c10::multiply_integers(x.sizes().slice(0, x.dim() - 1));
    expect_on_device_of(x, {&w1, &c1, &w2, &c2, &r}, "feed_forward");
    expect_epilogue(w1, c1, Tensor(), rows, "feed_forward");
    expect_epilogue(w2, c2, r, rows, "feed_forward");
    const c10::cuda::CUDAGuard on(x.device());
    if (wants_grad({&x, &w1, &c1, &w2, &c2, &r})) {
        return FeedForward::apply(x, w1, maybe(c1), w2, maybe(c2), maybe(r));
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    GemmExtra                                  e;
    e.bias         = bias_ready(c1);
    e.act          = 1;
    const Tensor x2 = rows_of(x, x.size(-1));
    e.out           = empty_operand(x2.size(0), w1.size(0), x);
    const Tensor h  = gemm(x2, w1, e);
    return linear_forward(h, w2, c2, r).view(shape_with_last(x.sizes(), w2.size(0)));
}

// ---- LayerNorm ---------------------------------------------------------------------------------------------
std::pair<Tensor, Tensor> layer_norm_forward(const Tensor& x2, double eps)
{
    const int64_t rows = x2.size(0), cols = x2.size(1);
    Tensor        y = empty_bf16({rows, cols}, x2), stats = empty_f32({rows, 2}, x2);
    ok(fu_layernorm_fwd(x2.data_ptr(), y.data_ptr(), static_cast<float*>(stats.data_ptr()), rows, cols, x2.stride(0), cols,
                        static_cast<float>(eps), stream_of(x2)));
    return {y, stats};
}

Tensor layer_norm_rows(const Tensor& x)
{
    Tensor x2 = rows_of(x, x.size(-1));
    if (x2.stride(1) != 1 || x2.stride(0) % 8 || reinterpret_cast<uintptr_t>(x2.data_ptr()) % 16) {
        x2 = x2.contiguous();
    }
    return x2;
}

Tensor layer_norm_backward(const Tensor& gy, const Tensor& x2, const Tensor& stats, const Tensor& add,
                           const std::vector<int64_t>& shape)
{
    const int64_t rows = x2.size(0), cols = x2.size(1);
    const Tensor  g2 = gy.reshape({rows, cols}).contiguous(), xc = x2.contiguous();
    Tensor        a2 = add.defined() ? aligned(add.reshape({rows, cols}).contiguous()) : add;
    Tensor        dx = empty_bf16({rows, cols}, gy);
    ok(fu_layernorm_bwd_add(g2.data_ptr(), xc.data_ptr(), static_cast<const float*>(stats.data_ptr()),
                            a2.defined() ? a2.data_ptr() : nullptr, dx.data_ptr(), rows, cols, cols, stream_of(gy)));
    return dx.view(shape);
}

struct LayerNorm : public torch::autograd::Function<LayerNorm> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, double eps)
    {
        const at::AutoDispatchBelowAutograd below;
        const Tensor x2        = layer_norm_rows(x);
        const auto [y, stats] = layer_norm_forward(x2, eps);
        ctx->save_for_backward({x2, stats});
        ctx->saved_data["shape"] = x.sizes().vec();
        return y.view(x.sizes());
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        const at::AutoDispatchBelowADInplaceOrView below;
        const variable_list        saved = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard on(saved[0].device());
        return {layer_norm_backward(grads[0], saved[0], saved[1], Tensor(), ctx->saved_data["shape"].toIntVector()), Tensor()};
    }
};

// LayerNorm in front of a residual branch: (norm(x), x). The gradient that comes back past the norm
// is added inside the norm's backward kernel instead of by a pass of its own.
struct LayerNormFork : public torch::autograd::Function<LayerNormFork> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, double eps)
    {
        const at::AutoDispatchBelowAutograd below;
        const Tensor x2        = layer_norm_rows(x);
        const auto [y, stats] = layer_norm_forward(x2, eps);
        ctx->save_for_backward({x2, stats});
        ctx->saved_data["shape"] = x.sizes().vec();
        ctx->set_materialize_grads(false);
        return {y.view(x.sizes()), x};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        const at::AutoDispatchBelowADInplaceOrView below;
        const variable_list saved = ctx->get_saved_variables();
        if (!grads[0].defined()) {
            return {grads[1], Tensor()};
        }
        const c10::cuda::CUDAGuard on(saved[0].device());
        return {layer_norm_backward(grads[0], saved[0], saved[1], grads[1], ctx->saved_data["shape"].toIntVector()), Tensor()};
    }
};

void check_norm(const Tensor& x)
{
    expect(x.scalar_type() == at::kBFloat16 && x.dim() >= 1 && x.size(-1) % 8 == 0, "layer_norm: bf16 rows of a multiple of 8 "
           "columns, got ", x.scalar_type(), " ", x.sizes());
}

Tensor layer_norm_entry(const Tensor& x, double eps)
{
    check_norm(x);
    const c10::cuda::CUDAGuard on(x.device());
    if (wants_grad({&x})) {
        return LayerNorm::apply(x, eps);
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    return layer_norm_forward(layer_norm_rows(x), eps).first.view(x.sizes());
}

std::pair<Tensor, Tensor> layer_norm_fork_entry(const Tensor& x, double eps)
{
    check_norm(x);
    const c10::cuda::CUDAGuard on(x.device());
    if (wants_grad({&x})) {
        const variable_list both = LayerNormFork::apply(x, eps);
        return {both[0], both[1]};
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    return {layer_norm_forward(layer_norm_rows(x), eps).first.view(x.sizes()), x};
}

// ---- attention -------------------------------------------------------------------------------------------------
void attention_operand(const Tensor& t)
{
    expect(t.dim() == 4 && t.size(3) == kHeadDim && t.stride(3) == 1 && t.scalar_type() == at::kBFloat16,
           "attention operands are (b, s, h, 128) bf16 with a dense last axis: got ", t.sizes(), " strides ", t.strides());
}

FuFmhaArgs attention_args(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, std::optional<double> scale)
{
    expect_on_device_of(q, {&k, &v, &o}, "attention");
    for (const Tensor* t : {&q, &k, &v, &o}) {
        attention_operand(*t);
    }
    expect(k.size(0) == q.size(0) && k.size(2) == q.size(2) && k.sizes() == v.sizes() && o.size(0) >= q.size(0)
               && o.size(1) >= q.size(1) && o.size(2) >= q.size(2),
           "attention: q ",
           q.sizes(), ", k ", k.sizes(), ", v ", v.sizes(), ", result ", o.sizes());
    FuFmhaArgs a{};
    a.q        = q.data_ptr();
    a.k        = k.data_ptr();
    a.v        = v.data_ptr();
    a.o        = o.data_ptr();
    a.batch    = static_cast<int32_t>(q.size(0));
    a.seq_q    = static_cast<int32_t>(q.size(1));
    a.heads    = static_cast<int32_t>(q.size(2));
    a.seq_kv   = static_cast<int32_t>(k.size(1));
    a.head_dim = static_cast<int32_t>(kHeadDim);
    a.q_row = q.stride(1), a.q_head = q.stride(2), a.q_batch = q.stride(0);
    a.k_row = k.stride(1), a.k_head = k.stride(2), a.k_batch = k.stride(0);
    a.v_row = v.stride(1), a.v_head = v.stride(2), a.v_batch = v.stride(0);
    a.o_row = o.stride(1), a.o_head = o.stride(2), a.o_batch = o.stride(0);
    a.scale = static_cast<float>(scale.has_value() ? *scale : 1.0 / std::sqrt(static_cast<double>(kHeadDim)));
    a.err   = error_ptr(q);
    return a;
}

std::pair<Tensor, Tensor> fmha_fwd(const Tensor& q, const Tensor& k, const Tensor& v, std::optional<double> scale,
                                   const MaybeTensor& out, int64_t ctas, int64_t flags, const MaybeTensor& trace)
{
    expect(q.dim() == 4 && q.size(3) == kHeadDim && k.sizes() == v.sizes() && k.dim() == 4 && k.size(0) == q.size(0)
               && k.size(2) == q.size(2),
           "fmha_fwd: q ", q.sizes(), ", k ", k.sizes(), ", v ", v.sizes());
    const c10::cuda::CUDAGuard on(q.device());
    Tensor                     o   = out.has_value() ? *out : empty_bf16(q.sizes(), q);
    Tensor                     lse = empty_f32({q.size(0), q.size(2), q.size(1)}, q);
    FuFmhaArgs                 a   = attention_args(q, k, v, o, scale);
    a.lse                          = static_cast<float*>(lse.data_ptr());
    a.ctas                         = static_cast<int32_t>(ctas);
    a.flags                        = static_cast<int32_t>(flags);
    if (trace.has_value()) {
        expect(trace->scalar_type() == at::kLong && trace->numel() >= 256 && trace->is_cuda(), "fmha_fwd: trace is int64[256]");
        a.trace = reinterpret_cast<uint64_t*>(trace->data_ptr());
    }
    ok(fu_fmha_fwd(&a, stream_of(q)));
    return {o, lse};
}

std::tuple<Tensor, Tensor, Tensor> fmha_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o_in,
                                            const Tensor& lse, const Tensor& do_in, std::optional<double> scale, int64_t ctas,
                                            const std::optional<std::vector<Tensor>>& out, bool deterministic,
                                            const MaybeTensor& trace)
{
    const c10::cuda::CUDAGuard on(q.device());
    const int64_t              b = q.size(0), sq = q.size(1), h = q.size(2);
    Tensor                     o = o_in, d_o = aligned(do_in);
    if (d_o.strides() != o.strides()) {
        d_o = d_o.contiguous();
        o   = o.contiguous();
    }
    expect_on_device_of(q, {&d_o, &lse}, "fmha_bwd");
    expect(d_o.sizes() == o.sizes() && d_o.scalar_type() == at::kBFloat16, "fmha_bwd: the gradient of a result of ", o.sizes(),
           " is ", d_o.scalar_type(), " ", d_o.sizes());
    expect(lse.scalar_type() == at::kFloat && lse.is_contiguous() && lse.numel() == b * h * sq, "fmha_bwd: lse is (b, h, sq) dense fp32, got ",
           lse.scalar_type(), " ", lse.sizes());
    Tensor dq, dk, dv;
    if (out.has_value()) {
        expect(out->size() == 3, "fmha_bwd: out is (dq, dk, dv)");
        dq = (*out)[0], dk = (*out)[1], dv = (*out)[2];
        expect_on_device_of(q, {&dq, &dk, &dv}, "fmha_bwd");
        expect(dq.is_contiguous() && dk.is_contiguous() && dv.is_contiguous(), "fmha_bwd: out tensors must be dense");
        expect(dq.sizes() == q.sizes() && dk.sizes() == k.sizes() && dv.sizes() == v.sizes() && dq.scalar_type() == at::kBFloat16
                   && dk.scalar_type() == at::kBFloat16 && dv.scalar_type() == at::kBFloat16,
               "fmha_bwd: out is bf16 shaped like q, k, v, got ", dq.sizes(), ", ", dk.sizes(), ", ", dv.sizes());
    }
    else {
        dq = empty_bf16(q.sizes(), q);
        dk = empty_bf16(k.sizes(), q);
        dv = empty_bf16(k.sizes(), q);
    }
    // the launcher addresses dq/dk/dv with the strides of q/k/v: hand it dense q/k/v
    const Tensor  qc = q.contiguous(), kc = k.contiguous(), vc = v.contiguous();
    const int64_t sq_pad = (sq + 127) / 128 * 128;
    FuFmhaArgs    a      = attention_args(qc, kc, vc, o, scale);
    const Tensor  stats  = empty_f32({2 * b * h * sq_pad}, q);
    Tensor        acc;
    if (!deterministic) {
        acc      = empty_f32({b, sq, h, kHeadDim}, q);
        a.dq_acc = static_cast<float*>(acc.data_ptr());
    }
    a.lse   = static_cast<float*>(lse.data_ptr());
    a.ctas  = static_cast<int32_t>(ctas);
    a.d_o   = d_o.data_ptr();
    a.dq    = dq.data_ptr();
    a.dk    = dk.data_ptr();
    a.dv    = dv.data_ptr();
    a.delta = static_cast<float*>(stats.data_ptr());
    a.flags = deterministic ? FU_FMHA_DETERMINISTIC : 0;
    if (trace.has_value()) {
        a.trace = reinterpret_cast<uint64_t*>(trace->data_ptr());
    }
    ok(fu_fmha_bwd(&a, stream_of(q)));
    return {dq, dk, dv};
}

struct Attention : public torch::autograd::Function<Attention> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, std::optional<double> scale)
    {
        const at::AutoDispatchBelowAutograd below;
        const auto [o, lse] = fmha_fwd(q, k, v, scale, std::nullopt, 0, 0, std::nullopt);
        ctx->save_for_backward({q, k, v, o, lse});
        if (scale.has_value()) {
            ctx->saved_data["scale"] = *scale;
        }
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        const at::AutoDispatchBelowADInplaceOrView below;
        const variable_list   s = ctx->get_saved_variables();
        std::optional<double> scale;
        if (ctx->saved_data.count("scale")) {
            scale = ctx->saved_data["scale"].toDouble();
        }
        const auto [dq, dk, dv] =
            fmha_bwd(s[0], s[1], s[2], s[3], s[4], grads[0].contiguous(), scale, 0, std::nullopt, false, std::nullopt);
        return {dq, dk, dv, Tensor()};
    }
};

Tensor attention_entry(const Tensor& q, const Tensor& k, const Tensor& v, std::optional<double> scale)
{
    if (wants_grad({&q, &k, &v})) {
        return Attention::apply(q, k, v, scale);
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    return fmha_fwd(q, k, v, scale, std::nullopt, 0, 0, std::nullopt).first;
}

// ---- the sequence-parallel attention block --------------------------------------------------------------------
// One per module: the geometry, the addresses of every rank's symmetric buffers and this rank's views
// of them. Python allocates the buffers (collectively) and keeps them alive beside this object.
struct SpAttention : public torch::CustomClassHolder {
    int64_t              heads, rank, world, s_local, seq_off, s_total, batch, region, timeout_ms;
    double               eps;
    std::vector<int64_t> head_splits;
    std::vector<int64_t> qkv_base, qkv_ctrl, o_base, o_ctrl, do_base, do_ctrl, dqkv_base, dqkv_ctrl;
    Tensor               q, k, v, o, d_o, dq, dk, dv;
    Tensor               ready;  // flags of the pull kernel, grown on demand
    int64_t              comm_stream = 0;  // the group's comm stream (0: none)
    int64_t              forwards    = 0;  // q, k, v and o belong to the latest forward
    // A norm weight as the kernels read it: dense fp32 that starts on 16 bytes (a slice of a flat parameter buffer may
    // start anywhere). Made anew for each call: a write through `.data` leaves no trace that a kept copy could be judged by.
    static Tensor f32(const Tensor& param)
    {
        const Tensor p = param.detach();
        return aligned(p.scalar_type() == at::kFloat && p.is_contiguous() ? p : p.to(at::kFloat).contiguous());
    }

    // How many CTAs a fused GEMM kernel of this block may take right now (0 = the whole device).
    //
    // The fused kernels are persistent, one CTA per SM, and their CTAs wait on peers; an
    // asynchronous exchange of the same group is a kernel of the same kind on another stream.
    // If one held every SM on this rank while the other could not start here, and the opposite
    // happened on a peer, each would wait for a kernel that cannot run. So while the group's comm
    // stream has work queued, a fused kernel leaves the SMs an asynchronous exchange takes (a
    // third of the device) free; with the comm stream idle it takes everything. All ranks issue
    // the same calls in the same order, so a rank that sees its comm stream idle has an exchange
    // that every peer has already been able to start.
    int64_t fused_ctas() const
    {
        if (world == 1 || comm_stream == 0) {
            return 0;
        }
        const cudaError_t state = cudaStreamQuery(reinterpret_cast<cudaStream_t>(comm_stream));
        if (state == cudaSuccess) {
            return 0;
        }
        TORCH_CHECK(state == cudaErrorNotReady, "fast_ulysses_b200: comm stream: ", cudaGetErrorString(state));
        const int64_t sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
        return sms - sms / 3;
    }

    void scatter(const Tensor& x2, const Tensor& w, const std::vector<int64_t>& base, const std::vector<int64_t>& ctrl,
                 int n_types, int n_normed, const Tensor& rope, const Tensor& gq, const Tensor& gk, const Tensor& y_save,
                 bool w_kn) const
    {
        expect(w.size(w_kn ? 1 : 0) == n_types * heads * kHeadDim && w.size(w_kn ? 0 : 1) == x2.size(1) && w.stride(1) == 1
                   && x2.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16,
               "attention block: activations ", x2.sizes(), " x weight ", w.sizes());
        FuQkvArgs a{};
        a.x = x2.data_ptr();
        a.w = w.data_ptr();
        a.m = x2.size(0);
        a.k = x2.size(1);
        a.ldx = x2.stride(0);
        a.ldw = w.stride(0);
        a.flags = w_kn ? FU_QKV_W_KN : 0;
        a.heads = static_cast<int32_t>(heads);
        a.s_local = s_local;
        a.seq_off = seq_off;
        a.s_total = s_total;
        a.eps     = static_cast<float>(eps);
        a.rank    = static_cast<int32_t>(rank);
        a.world   = static_cast<int32_t>(world);
        if (n_normed) {
            a.rope    = static_cast<const float*>(rope.data_ptr());
            a.gamma_q = static_cast<const float*>(gq.data_ptr());
            a.gamma_k = static_cast<const float*>(gk.data_ptr());
        }
        for (int64_t p = 0; p < world; ++p) {
            a.head_splits[p] = static_cast<int32_t>(head_splits[p]);
            a.win_q[p]       = reinterpret_cast<void*>(base[p]);
            a.win_k[p]       = reinterpret_cast<void*>(base[p] + region);
            a.win_v[p]       = reinterpret_cast<void*>(base[p] + 2 * region);
            a.peer_ctrl[p]   = reinterpret_cast<FuCtrl*>(ctrl[p]);
        }
        a.timeout_ms = static_cast<uint32_t>(timeout_ms);
        a.ctas       = static_cast<int32_t>(fused_ctas());
        a.err        = error_ptr(x2);
        a.n_types    = n_types;
        a.n_normed   = n_normed;
        a.win_bytes  = region;
        if (y_save.defined()) {
            a.y_save = y_save.data_ptr();
            a.ld_y   = y_save.stride(0);
        }
        ok(fu_qkv_rope_scatter(&a, stream_of(x2)));
    }

    // A operand pulled from the owners of the heads; returns (result, gathered operand).
    std::pair<Tensor, Tensor> pull_outproj(const Tensor& w, const Tensor& bias, const Tensor& residual)
    {
        const int64_t m = batch * s_local, hidden = w.size(0);
        expect(w.dim() == 2 && w.size(1) == heads * kHeadDim && w.stride(1) == 1 && w.scalar_type() == at::kBFloat16,
               "attention block: output weight ", w.sizes());
        if (world == 1) {
            // Nothing to pull: this rank's attention output is the operand as it lies in its buffer (which
            // stays this forward's until the next forward, like q, k and v).
            GemmExtra e;
            e.bias         = bias_ready(bias);
            e.residual     = residual;
            const Tensor a = o.view({m, heads * kHeadDim});
            return {gemm(a, w, e), a};
        }
        Tensor        gather = empty_bf16({m, heads * kHeadDim}, w), out = empty_bf16({m, hidden}, w);
        const int64_t flags = (m + 127) / 128 * world;
        if (!ready.defined() || ready.numel() < flags) {
            ready = at::zeros({flags}, at::TensorOptions().dtype(at::kInt).device(w.device()));
        }
        FuPullArgs a{};
        a.w   = w.data_ptr();
        a.c   = out.data_ptr();
        a.m   = m;
        a.n   = hidden;
        a.ldw = w.stride(0);
        a.ldc = hidden;
        const Tensor b = bias_ready(bias);
        if (b.defined()) {
            a.bias = b.data_ptr();
            a.flags |= b.scalar_type() == at::kBFloat16 ? FU_PULL_BIAS_BF16 : 0;
        }
        a.residual = residual.defined() ? residual.data_ptr() : nullptr;
        a.s_local  = s_local;
        a.seq_off  = seq_off;
        a.s_total  = s_total;
        a.rank     = static_cast<int32_t>(rank);
        a.world    = static_cast<int32_t>(world);
        for (int64_t p = 0; p < world; ++p) {
            a.head_splits[p] = static_cast<int32_t>(head_splits[p]);
            a.peer_o[p]      = reinterpret_cast<const void*>(o_base[p]);
            a.peer_ctrl[p]   = reinterpret_cast<FuCtrl*>(o_ctrl[p]);
        }
        a.gather       = gather.data_ptr();
        a.ready        = static_cast<uint32_t*>(ready.data_ptr());
        a.o_bytes      = region;
        a.gather_bytes = gather.numel() * 2;
        a.ready_words  = ready.numel();
        a.timeout_ms   = static_cast<uint32_t>(timeout_ms);
        a.ctas         = static_cast<int32_t>(fused_ctas());
        a.err          = error_ptr(w);
        ok(fu_pull_outproj(&a, stream_of(w)));
        return {out, gather};
    }

    struct Forward {
        Tensor out, x2, y_save, gather, lse;
    };

    Forward forward(const Tensor& x, const Tensor& w_qkv, const Tensor& gamma_q, const Tensor& gamma_k, const Tensor& w_o,
                    const Tensor& b_o, const Tensor& residual, const Tensor& rope, bool need_grad)
    {
        const int64_t m = batch * s_local, hidden = x.size(-1);
        Forward       f;
        f.x2 = x.reshape({m, hidden});
        if (f.x2.stride(1) != 1 || f.x2.stride(0) % 8) {
            f.x2 = f.x2.contiguous();
        }
        ++forwards;
        if (need_grad) {
            f.y_save = empty_bf16({m, 2 * heads * kHeadDim}, x);
        }
        {
            const NvtxRange r("fast_ulysses_b200::qkv_norm_rope_scatter");
            scatter(f.x2, w_qkv, qkv_base, qkv_ctrl, 3, 2, rope, f32(gamma_q), f32(gamma_k), f.y_save, false);
        }
        {
            const NvtxRange r("fast_ulysses_b200::fmha_fwd");
            f.lse = fmha_fwd(q, k, v, std::nullopt, o, 0, 0, std::nullopt).second;
        }
        const NvtxRange r("fast_ulysses_b200::pull_outproj");
        std::tie(f.out, f.gather) =
            pull_outproj(w_o, b_o, residual.defined() ? aligned(residual.reshape({m, hidden}).contiguous()) : residual);
        f.out = f.out.view(x.sizes());
        return f;
    }
};

using SpPtr = c10::intrusive_ptr<SpAttention>;

struct SpAttentionFn : public torch::autograd::Function<SpAttentionFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w_qkv, const Tensor& gamma_q,
                          const Tensor& gamma_k, const Tensor& w_o, const MaybeTensor& b_o, const MaybeTensor& residual,
                          const Tensor& rope, const SpPtr& mod)
    {
        const at::AutoDispatchBelowAutograd below;
        const auto f = mod->forward(x, w_qkv, gamma_q, gamma_k, w_o, or_none(b_o), or_none(residual), rope, true);
        ctx->saved_data["b_o"]      = b_o.has_value();
        ctx->saved_data["residual"] = residual.has_value();
        ctx->save_for_backward({f.x2, w_qkv, gamma_q, gamma_k, w_o, f.y_save, f.gather, f.lse, rope});
        ctx->saved_data["mod"]     = c10::IValue::make_capsule(mod);
        ctx->saved_data["forward"] = mod->forwards;
        ctx->saved_data["x_shape"] = x.sizes().vec();
        return f.out;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        const at::AutoDispatchBelowADInplaceOrView below;
        const variable_list s = ctx->get_saved_variables();
        const Tensor        x2 = s[0], w_qkv = s[1], gamma_q = s[2], gamma_k = s[3], w_o = s[4], y_save = s[5], gather = s[6],
                     lse = s[7], rope = s[8], dy = grads[0];
        const SpPtr   mod = c10::static_intrusive_pointer_cast<SpAttention>(ctx->saved_data["mod"].toCapsule());
        const int64_t mine = ctx->saved_data["forward"].toInt();
        TORCH_CHECK(mine == mod->forwards,
                    "UlyssesSelfAttention: forward ran again on this module before this backward; q, k, v and the attention "
                    "output live in the module's symmetric buffers and now belong to the later call (this backward is for "
                    "forward #", mine, ", the buffers hold #", mod->forwards,
                    "). Run backward before the next forward (gradient accumulation: forward, backward, forward, backward), use "
                    "one module per activation that must stay alive, or recompute the forward.");
        const c10::cuda::CUDAGuard on(dy.device());
        const std::vector<int64_t> shape = ctx->saved_data["x_shape"].toIntVector();
        const int64_t              hidden = shape.back(), m = mod->batch * mod->s_local, heads = mod->heads;
        const Tensor               dy2 = dy.reshape({m, hidden}).contiguous();
        variable_list              out(9);
        const Wanted wanted(ctx, {true, true, true, true, true, ctx->saved_data["b_o"].toBool(),
                                  ctx->saved_data["residual"].toBool()});
        GemmExtra                  wgrad;
        wgrad.a_km = wgrad.b_kn = true;
        if (wanted[5]) {
            out[5] = column_sum(dy2);
        }
        if (wanted[4]) {
            out[4] = gemm(dy2, gather, wgrad);  // dW_o[n, k] = sum_m dy[m, n] A[m, k]
        }
        if (wanted[6]) {
            out[6] = dy;
        }
        // dA = dy W_o, scattered to the head owners from the GEMM epilogue (mode-0 direction); W_o is
        // (hidden, heads * 128) = (contraction, output) as stored, so nothing is transposed
        {
            const NvtxRange r("fast_ulysses_b200::dout_scatter");
            mod->scatter(dy2, w_o, mod->do_base, mod->do_ctrl, 1, 0, Tensor(), Tensor(), Tensor(), Tensor(), true);
        }
        {
            const NvtxRange r("fast_ulysses_b200::fmha_bwd");
            fmha_bwd(mod->q, mod->k, mod->v, mod->o, lse, mod->d_o, std::nullopt, 0,
                     std::vector<Tensor>{mod->dq, mod->dk, mod->dv}, false, std::nullopt);
        }
        // dq, dk, dv come home inside the kernel that undoes RoPE and RMSNorm (mode-1 direction)
        const Tensor dyqkv = empty_bf16({m, 3 * heads * kHeadDim}, dy);
        const Tensor dg    = empty_f32({2, kHeadDim}, dy);
        C10_CUDA_CHECK(cudaMemsetAsync(dg.data_ptr(), 0, dg.nbytes(), stream_of(dy)));
        {
            const NvtxRange r("fast_ulysses_b200::pull_qkv_grads");
            const Tensor    gq = SpAttention::f32(gamma_q), gk = SpAttention::f32(gamma_k);
            FuPullGradsArgs a{};
            for (int64_t p = 0; p < mod->world; ++p) {
                a.peer_dq[p]     = reinterpret_cast<const void*>(mod->dqkv_base[p]);
                a.peer_dk[p]     = reinterpret_cast<const void*>(mod->dqkv_base[p] + mod->region);
                a.peer_dv[p]     = reinterpret_cast<const void*>(mod->dqkv_base[p] + 2 * mod->region);
                a.peer_ctrl[p]   = reinterpret_cast<FuCtrl*>(mod->dqkv_ctrl[p]);
                a.head_splits[p] = static_cast<int32_t>(mod->head_splits[p]);
            }
            a.src_bytes  = mod->region;
            a.y          = y_save.data_ptr();
            a.dy         = dyqkv.data_ptr();
            a.rope       = static_cast<const float*>(rope.data_ptr());
            a.gamma_q    = static_cast<const float*>(gq.data_ptr());
            a.gamma_k    = static_cast<const float*>(gk.data_ptr());
            a.dgamma_q   = static_cast<float*>(dg.data_ptr());
            a.dgamma_k   = static_cast<float*>(dg.data_ptr()) + kHeadDim;
            a.m          = m;
            a.s_local    = mod->s_local;
            a.seq_off    = mod->seq_off;
            a.s_total    = mod->s_total;
            a.ld_y       = y_save.stride(0);
            a.ld_dy      = dyqkv.stride(0);
            a.heads      = static_cast<int32_t>(heads);
            a.rank       = static_cast<int32_t>(mod->rank);
            a.world      = static_cast<int32_t>(mod->world);
            a.timeout_ms = static_cast<uint32_t>(mod->timeout_ms);
            a.eps        = static_cast<float>(mod->eps);
            ok(fu_pull_qkv_grads(&a, stream_of(dy)));
        }
        if (wanted[0]) {
            GemmExtra e;
            e.b_kn = true;
            out[0] = gemm(dyqkv, w_qkv, e).view(shape);
        }
        if (wanted[1]) {
            out[1] = gemm(dyqkv, x2, wgrad);
        }
        if (wanted[2]) {
            out[2] = as_type_of(dg[0], gamma_q);
        }
        if (wanted[3]) {
            out[3] = as_type_of(dg[1], gamma_k);
        }
        return out;
    }
};

Tensor sp_attention_entry(const SpPtr& mod, const Tensor& x, const Tensor& w_qkv, const Tensor& gamma_q, const Tensor& gamma_k,
                          const Tensor& w_o, const MaybeTensor& b_o, const MaybeTensor& residual, const Tensor& rope)
{
    expect(x.dim() == 3 && x.size(0) == mod->batch && x.size(1) == mod->s_local && x.scalar_type() == at::kBFloat16,
           "UlyssesSelfAttention: input ", x.scalar_type(), " ", x.sizes(), ", expected bf16 (", mod->batch, ", ", mod->s_local,
           ", hidden)");
    const Tensor r = or_none(residual), b = or_none(b_o);
    expect(!r.defined() || (r.sizes() == x.sizes() && r.scalar_type() == at::kBFloat16),
           "UlyssesSelfAttention: the residual must be bf16 and shaped like the input");
    expect_on_device_of(x, {&w_qkv, &gamma_q, &gamma_k, &w_o, &b, &r, &rope}, "UlyssesSelfAttention");
    expect(gamma_q.numel() == kHeadDim && gamma_k.numel() == kHeadDim && rope.is_contiguous() && rope.scalar_type() == at::kFloat
               && rope.numel() == mod->s_local * kHeadDim,
           "UlyssesSelfAttention: norm weights of ", kHeadDim, " values and a dense fp32 table of ", mod->s_local, " positions, got ",
           gamma_q.sizes(), ", ", gamma_k.sizes(), " and ", rope.sizes());
    expect(w_o.dim() == 2, "UlyssesSelfAttention: output weight ", w_o.sizes());
    expect_epilogue(w_o, b, r, mod->batch * mod->s_local, "UlyssesSelfAttention");
    const c10::cuda::CUDAGuard on(x.device());
    if (wants_grad({&x, &w_qkv, &gamma_q, &gamma_k, &w_o, &b, &r})) {
        return SpAttentionFn::apply(x, w_qkv, gamma_q, gamma_k, w_o, maybe(b), maybe(r), rope, mod);
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    return mod->forward(x, w_qkv, gamma_q, gamma_k, w_o, b, r, rope, false).out;
}

// ---- block-scaled fp8 exchange ----------------------------------------------------------------------------------
Tensor fp8_exchange(const GroupRef& ref, const Tensor& x_in, int64_t mode, const Splits& seq, const Splits& heads)
{
    Group& g = *ref.group;
    expect(x_in.dim() == 4 && x_in.size(3) == kHeadDim && x_in.scalar_type() == at::kBFloat16,
           "all_to_all_4d_fp8: (b, s, n, 128) bf16, got ", x_in.scalar_type(), " ", x_in.sizes());
    g.check_alive();
    const c10::cuda::CUDAGuard                 on(x_in.device());
    const at::AutoDispatchBelowADInplaceOrView below;
    Tensor                                     x    = x_in.contiguous();
    const std::shared_ptr<const Plan>          kept = g.plan(x.sizes(), {}, x.scalar_type(), mode, seq, heads);
    const Plan&                                plan = *kept;
    Tensor                                     out  = empty_bf16(plan.out_shape, x);
    const int                                  world = g.world(), rank = g.rank();
    if (world == 1) {
        if (reinterpret_cast<uintptr_t>(x.data_ptr()) % 32) {
            x = x.clone();
        }
        ok(fu_fp8_round_trip(x.data_ptr(), out.data_ptr(), x.numel() / kHeadDim, stream_of(x)));
        return out;
    }
    constexpr int64_t kPacked = 144;  // bytes of a packed row: 128 payload, scale, padding
    const int64_t     win_bytes = plan.window_numel / kHeadDim * kPacked;  // the largest result of any rank, packed
    // one symmetric window per group, grown collectively (every rank computes the same size)
    const Window& w = g.window(Role::kFp8, win_bytes);
    FuA2AFp8Args  a{};
    a.src = x.data_ptr();
    a.out = out.data_ptr();
    for (int p = 0; p < world; ++p) {
        a.peer_win[p]  = w.base[p];
        a.peer_ctrl[p] = w.ctrl[p];
    }
    a.win_bytes = w.capacity;
    a.src_bytes = x.numel() * 2;
    a.out_rows  = out.numel() / kHeadDim;
    a.rank      = rank;
    a.world     = world;
    // start with the next rank up, as the bf16 exchange does, so every rank's ingress has one sender at a time
    for (int i = 1; i <= world; ++i) {
        for (const Route& r : plan.sends) {
            if (r.peer == (rank + i) % world) {
                a.routes[a.n_routes++] = FuRoute{r.peer, 0, r.src_off, r.dst_off, r.src_pitch, r.dst_pitch, r.row_bytes, r.rows,
                                                 r.batches, r.src_batch, r.dst_batch};
            }
        }
    }
    a.flags      = g.test_flags();
    a.timeout_ms = g.timeout_ms();
    ok(fu_a2a4d_fp8(&a, stream_of(x)));
    return out;
}

}  // namespace

void bind_fused(py::module_& m)
{
    m.def("error_word", &error_word);
    m.def("gemm_bf16", torch::wrap_pybind_function_no_gil(&gemm_entry));
    m.def("linear", torch::wrap_pybind_function_no_gil(&linear_entry));
    m.def("feed_forward", torch::wrap_pybind_function_no_gil(&feed_forward_entry));
    m.def("layer_norm", torch::wrap_pybind_function_no_gil(&layer_norm_entry));
    m.def("layer_norm_fork", torch::wrap_pybind_function_no_gil(&layer_norm_fork_entry));
    m.def("fmha_fwd", torch::wrap_pybind_function_no_gil(&fmha_fwd));
    m.def("fmha_bwd", torch::wrap_pybind_function_no_gil(&fmha_bwd));
    m.def("attention", torch::wrap_pybind_function_no_gil(&attention_entry));
    m.def("fp8_exchange", torch::wrap_pybind_function_no_gil(&fp8_exchange));
    py::class_<SpAttention, SpPtr>(m, "SpAttention")
        .def(py::init([]() { return c10::make_intrusive<SpAttention>(); }))
        .def_readwrite("heads", &SpAttention::heads)
        .def_readwrite("rank", &SpAttention::rank)
        .def_readwrite("world", &SpAttention::world)
        .def_readwrite("s_local", &SpAttention::s_local)
        .def_readwrite("seq_off", &SpAttention::seq_off)
        .def_readwrite("s_total", &SpAttention::s_total)
        .def_readwrite("batch", &SpAttention::batch)
        .def_readwrite("region", &SpAttention::region)
        .def_readwrite("timeout_ms", &SpAttention::timeout_ms)
        .def_readwrite("eps", &SpAttention::eps)
        .def_readwrite("head_splits", &SpAttention::head_splits)
        .def_readwrite("comm_stream", &SpAttention::comm_stream)
        .def_readonly("forwards", &SpAttention::forwards)
        .def("set_buffers",
             [](SpAttention& s, const std::vector<std::vector<int64_t>>& addresses, const std::vector<Tensor>& views) {
                 TORCH_CHECK(addresses.size() == 8 && views.size() == 8, "SpAttention: four buffers (base, ctrl) and eight views");
                 s.qkv_base = addresses[0], s.qkv_ctrl = addresses[1], s.o_base = addresses[2], s.o_ctrl = addresses[3];
                 s.do_base = addresses[4], s.do_ctrl = addresses[5], s.dqkv_base = addresses[6], s.dqkv_ctrl = addresses[7];
                 s.q = views[0], s.k = views[1], s.v = views[2], s.o = views[3];
                 s.d_o = views[4], s.dq = views[5], s.dk = views[6], s.dv = views[7];
             })
        // the two scatters and the pull on their own, for benchmarks of single kernels
        .def("scatter_qkv",
             [](SpAttention& s, const Tensor& x2, const Tensor& w, const Tensor& rope, const Tensor& gq, const Tensor& gk,
                const MaybeTensor& y_save) {
                 s.scatter(x2, w, s.qkv_base, s.qkv_ctrl, 3, 2, rope, SpAttention::f32(gq),
                           SpAttention::f32(gk), or_none(y_save), false);
             })
        .def("scatter_dout",
             [](SpAttention& s, const Tensor& dy2, const Tensor& w_o) {
                 s.scatter(dy2, w_o, s.do_base, s.do_ctrl, 1, 0, Tensor(), Tensor(), Tensor(), Tensor(), true);
             })
        .def("pull_outproj", [](SpAttention& s, const Tensor& w_o) { return s.pull_outproj(w_o, Tensor(), Tensor()); });
    m.def("sp_attention", torch::wrap_pybind_function_no_gil(&sp_attention_entry));
}

}  // namespace fu
