// Native tensor front end of the C ABI (include/o1d.h): argument checks, output and workspace allocation
// through torch's caching allocator, device guard, stream, and the call, in one crossing from Python.  The
// same steps written in Python around ctypes cost 40-60 us a call, several times the kernel at small sizes.
//
// Parameters (weights, biases, LayerNorm scales) are passed as they are stored when the kernels take bf16
// ones (O1D_FLAG_PARAMS_BF16); otherwise, or when the library has no such kernel for the request, they are
// converted to fp32 first.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../../include/o1d.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

py::object *g_check = nullptr;               // _lib.check(status, what): raises

void check(int status, const char *what) {
    if (status == O1D_OK) return;
    py::gil_scoped_acquire gil;
    (*g_check)(status, what);
}

int dtype_code(const Tensor &t) {
    if (t.scalar_type() == at::kFloat) return O1D_F32;
    if (t.scalar_type() == at::kBFloat16) return O1D_BF16;
    throw py::type_error("oriented1d_b200 supports float32 and bfloat16 tensors, got torch." + std::string(c10::toString(t.scalar_type())));
}
void need_cuda(const Tensor &t) {
    if (!t.is_cuda()) throw std::runtime_error("tensor must be a CUDA tensor (oriented1d_b200 has no CPU path)");
}
void need_cuda(const OptTensor &t) { if (t) need_cuda(*t); }
Tensor as_f32(const Tensor &t) { return t.detach().to(at::kFloat).contiguous(); }
bool is_bf16(const Tensor &t) { return t.scalar_type() == at::kBFloat16; }
void *stream() { return at::cuda::getCurrentCUDAStream().stream(); }
const void *ptr(const Tensor &t) { return t.defined() ? t.const_data_ptr() : nullptr; }

// Parameters as the library takes them: the stored bf16 values, or fp32 copies.
struct Params {
    Tensor w, b;
    bool bf16;
    Params(const Tensor &w_, const OptTensor &b_) : bf16(is_bf16(w_) && (!b_ || is_bf16(*b_))) {
        w = w_.contiguous();
        if (b_) b = b_->contiguous();
        if (!bf16) widen();
    }
    void widen() {
        w = as_f32(w);
        if (b.defined()) b = as_f32(b);
        bf16 = false;
    }
    int flag() const { return bf16 ? O1D_FLAG_PARAMS_BF16 : 0; }
};
// f(flag) with the parameters as stored, and again with fp32 ones where the library declines those.
template <class F> void call(Params &p, const char *what, F &&f) {
    int rc = f(p.flag());
    if (rc == O1D_ERR_UNSUPPORTED && p.bf16) {
        p.widen();
        rc = f(0);
    }
    check(rc, what);
}

struct Dims { int64_t n, h, w, c; };
Dims dims(const Tensor &t, bool nhwc) {
    if (t.dim() != 4) throw py::value_error("expected a 4-D tensor");
    return nhwc ? Dims{t.size(0), t.size(1), t.size(2), t.size(3)} : Dims{t.size(0), t.size(2), t.size(3), t.size(1)};
}
void check_params(int64_t plan_c, int64_t K, int64_t C, const Tensor *w, const OptTensor *bias) {
    // the kernels index w as [C, K] and bias as [C]: a shorter buffer would be read past its end
    if (plan_c != C)
        throw py::value_error("plan was built for " + std::to_string(plan_c) + " channels, tensor has " + std::to_string(C));
    if (w && w->numel() != C * K)
        throw py::value_error("weight has " + std::to_string(w->numel()) + " elements, expected C*K = " + std::to_string(C * K));
    if (bias && *bias && (*bias)->numel() != C)
        throw py::value_error("bias has " + std::to_string((*bias)->numel()) + " elements, expected C = " + std::to_string(C));
}
// Extents of an output are divided by the stride before the library sees it.
void need_stride(int64_t stride) {
    if (stride <= 0) throw py::value_error("stride must be positive, got " + std::to_string(stride));
}
std::vector<int64_t> shape(int64_t n, int64_t h, int64_t w, int64_t c, bool nhwc) {
    return nhwc ? std::vector<int64_t>{n, h, w, c} : std::vector<int64_t>{n, c, h, w};
}

Tensor fprop(const Tensor &x_, const Tensor &w, const OptTensor &bias, int64_t plan_c, int64_t K, int64_t host, int64_t dev,
             int64_t stride, bool nhwc, bool identity, bool gelu) {
    const Dims d = dims(x_, nhwc);
    need_stride(stride);
    check_params(plan_c, K, d.c, &w, &bias);
    need_cuda(x_); need_cuda(w); need_cuda(bias);
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = x_.contiguous();
    const int code = dtype_code(x);
    Params p(w, bias);
    Tensor y = at::empty(shape(d.n, (d.h + stride - 1) / stride, (d.w + stride - 1) / stride, d.c, nhwc), x.options());
    const int flags = (identity ? O1D_FLAG_IDENTITY : 0) | (gelu ? O1D_FLAG_GELU_INPUT : 0);
    void *out = y.data_ptr(), *st = stream();
    call(p, "o1d_fprop", [&](int pf) {
        return o1d_fprop(ptr(x), (const float *)ptr(p.w), (const float *)ptr(p.b), (const void *)host, (const void *)dev, out, (int)d.n,
                         (int)d.h, (int)d.w, (int)d.c, (int)K, (int)stride, nhwc, code, flags | pf | O1D_FLAG_MAY_CONVERT, st);
    });
    return y;
}

Tensor dgrad(const Tensor &dy_, const Tensor &w, int64_t plan_c, int64_t K, int64_t host, int64_t dev, int64_t H, int64_t W,
             int64_t stride, bool nhwc, bool identity, const OptTensor &pre_) {
    const Dims d = dims(dy_, nhwc);
    need_stride(stride);
    if (d.h != (H + stride - 1) / stride || d.w != (W + stride - 1) / stride)
        throw py::value_error("dy extents do not match ceil(H/stride) x ceil(W/stride)");
    check_params(plan_c, K, d.c, &w, nullptr);
    need_cuda(dy_); need_cuda(w);
    const c10::cuda::CUDAGuard guard(dy_.device());
    const Tensor dy = dy_.contiguous();
    const int code = dtype_code(dy);
    Params p(w, std::nullopt);
    Tensor dx = at::empty(shape(d.n, H, W, d.c, nhwc), dy.options()), pre;
    if (pre_) {
        if (pre_->sizes() != dx.sizes() || pre_->scalar_type() != dy.scalar_type())
            throw py::value_error("pre must have the shape and dtype of dx");
        need_cuda(*pre_);
        pre = pre_->contiguous();
    }
    void *out = dx.data_ptr(), *st = stream();
    call(p, "o1d_dgrad", [&](int pf) {
        return o1d_dgrad_act(ptr(dy), (const float *)ptr(p.w), ptr(pre), (const void *)host, (const void *)dev, out, (int)d.n, (int)H,
                             (int)W, (int)d.c, (int)K, (int)stride, nhwc, code, (identity ? O1D_FLAG_IDENTITY : 0) | pf | O1D_FLAG_MAY_CONVERT, st);
    });
    return dx;
}

// dw [C,1,1,K] and db [C] (or None), in fp32, or in bf16 when `bf16` is set.
std::tuple<Tensor, OptTensor> wgrad(const Tensor &dy_, const Tensor &x_, int64_t plan_c, int64_t K, int64_t host, int64_t dev,
                                    int64_t stride, bool nhwc, bool with_bias, bool gelu, bool bf16) {
    if (dy_.scalar_type() != x_.scalar_type()) throw py::type_error("dy and x must have the same dtype");
    const Dims d = dims(x_, nhwc);
    need_stride(stride);
    check_params(plan_c, K, d.c, nullptr, nullptr);
    const auto want = shape(d.n, (d.h + stride - 1) / stride, (d.w + stride - 1) / stride, d.c, nhwc);
    if (dy_.sizes() != at::IntArrayRef(want)) {
        std::ostringstream s;
        s << "dy has shape " << dy_.sizes() << ", expected the output shape of x (" << at::IntArrayRef(want) << ")";
        throw py::value_error(s.str());
    }
    need_cuda(dy_); need_cuda(x_);
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor dy = dy_.contiguous(), x = x_.contiguous();
    const int code = dtype_code(x);
    auto opts = x.options().dtype(bf16 ? at::kBFloat16 : at::kFloat);
    Tensor dw = at::empty({d.c, 1, 1, K}, opts), db;
    if (with_bias) db = at::empty({d.c}, opts);
    const size_t bytes = std::max<size_t>(16, o1d_wgrad_workspace_bytes((int)d.n, (int)d.h, (int)d.w, (int)d.c, (int)K, (int)stride, nhwc, code));
    Tensor ws = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
    void *st = stream();
    auto run = [&](int flag) {
        return o1d_wgrad_act(ptr(dy), ptr(x), (const void *)host, (const void *)dev, (float *)dw.data_ptr(),
                             with_bias ? (float *)db.data_ptr() : nullptr, ws.data_ptr(), bytes, (int)d.n, (int)d.h, (int)d.w, (int)d.c,
                             (int)K, (int)stride, nhwc, code, (gelu ? O1D_FLAG_GELU_INPUT : 0) | flag | O1D_FLAG_MAY_CONVERT, st);
    };
    int rc = run(bf16 ? O1D_FLAG_PARAMS_BF16 : 0);
    if (rc == O1D_ERR_UNSUPPORTED && bf16) {             // kernels that write fp32 gradients only
        dw = at::empty({d.c, 1, 1, K}, x.options().dtype(at::kFloat));
        if (with_bias) db = at::empty({d.c}, x.options().dtype(at::kFloat));
        rc = run(0);
        if (rc == O1D_OK) {
            dw = dw.to(at::kBFloat16);
            if (with_bias) db = db.to(at::kBFloat16);
        }
    }
    check(rc, "o1d_wgrad");
    return {dw, with_bias ? OptTensor(db) : std::nullopt};
}

Tensor transpose(const Tensor &t_, bool to_nhwc) {
    need_cuda(t_);
    if (t_.dim() != 4) throw py::value_error("expected a 4-D tensor");
    const c10::cuda::CUDAGuard guard(t_.device());
    const Tensor t = t_.contiguous();
    const int code = dtype_code(t);
    const int64_t n = t.size(0), hw = to_nhwc ? t.size(2) * t.size(3) : t.size(1) * t.size(2), c = to_nhwc ? t.size(1) : t.size(3);
    Tensor out = to_nhwc ? at::empty({n, t.size(2), t.size(3), c}, t.options()) : at::empty({n, c, t.size(1), t.size(2)}, t.options());
    check(o1d_transpose(ptr(t), out.data_ptr(), (int)n, (int)(to_nhwc ? c : hw), (int)(to_nhwc ? hw : c), code, stream()), "o1d_transpose");
    return out;
}

// The kernels read `expected` elements of a parameter: a shorter buffer would be read past its end.
void need_numel(const Tensor &t, int64_t expected, const char *what) {
    if (t.numel() != expected)
        throw py::value_error(std::string(what) + " has " + std::to_string(t.numel()) + " elements, expected " + std::to_string(expected));
}
// Length of the last axis of a tensor that is normalised or summed by rows.
int64_t row_length(const Tensor &x) {
    if (x.dim() == 0 || x.numel() == 0) throw py::value_error("expected a tensor with at least one row");
    return x.size(-1);
}

Tensor layer_norm_cl(const Tensor &x_, const Tensor &g, const Tensor &b, double eps, bool gelu) {
    need_numel(g, row_length(x_), "weight");
    need_numel(b, row_length(x_), "bias");
    need_cuda(x_); need_cuda(g); need_cuda(b);
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = x_.contiguous();
    const int code = dtype_code(x);
    const int64_t C = x.size(-1);
    Params p(g, b);
    Tensor y = at::empty_like(x);
    void *st = stream();
    call(p, "o1d_layernorm_cl", [&](int pf) {
        return o1d_layernorm_cl(ptr(x), (const float *)ptr(p.w), (const float *)ptr(p.b), y.data_ptr(), x.numel() / C, (int)C, (float)eps,
                                code, (gelu ? 1 : 0) | pf, st);
    });
    return y;
}

// dx, dweight, dbias; the last two in fp32, or in the parameters' dtype when `as_params` is set.
std::tuple<Tensor, Tensor, Tensor> layer_norm_cl_bwd(const Tensor &x_, const Tensor &dy_, const Tensor &g, double eps, const OptTensor &b,
                                                     bool gelu, bool as_params) {
    if (dy_.sizes() != x_.sizes() || dy_.scalar_type() != x_.scalar_type()) {
        std::ostringstream s;
        s << "dy " << dy_.sizes() << " " << dy_.scalar_type() << " does not match x " << x_.sizes() << " " << x_.scalar_type();
        throw py::value_error(s.str());
    }
    const int64_t C = row_length(x_), rows = x_.numel() / C;
    need_numel(g, C, "weight");
    if (gelu && (!b || b->numel() != C)) throw py::value_error("gelu=True needs the forward call's bias");
    need_cuda(x_); need_cuda(dy_); need_cuda(g);
    if (gelu) need_cuda(b);
    const Tensor x = x_.contiguous(), dy = dy_.contiguous();
    const c10::cuda::CUDAGuard guard(x.device());
    const int code = dtype_code(x);
    Params p(g, gelu ? b : OptTensor());
    const bool out_bf16 = as_params && p.bf16;
    if (!out_bf16 && p.bf16) p.widen();
    Tensor dx = at::empty_like(x);
    auto opts = x.options().dtype(out_bf16 ? at::kBFloat16 : at::kFloat);
    Tensor dg = at::empty({C}, opts), db = at::empty({C}, opts);
    const size_t bytes = o1d_layernorm_cl_bwd_workspace_bytes(rows, (int)C);
    Tensor ws = at::empty({(int64_t)std::max<size_t>(bytes, 4)}, x.options().dtype(at::kByte));
    check(o1d_layernorm_cl_bwd(ptr(x), ptr(dy), (const float *)ptr(p.w), (const float *)ptr(p.b), dx.data_ptr(), (float *)dg.data_ptr(),
                               (float *)db.data_ptr(), ws.data_ptr(), bytes, rows, (int)C, (float)eps, code,
                               (gelu ? 1 : 0) | (out_bf16 ? O1D_FLAG_PARAMS_BF16 : 0), stream()),
          "o1d_layernorm_cl_bwd");
    if (as_params && !out_bf16) { dg = dg.to(g.scalar_type()); db = db.to(b ? b->scalar_type() : g.scalar_type()); }
    return {dx, dg, db};
}

Tensor colsum(const Tensor &x_, bool bf16) {
    const int64_t C = row_length(x_), rows = x_.numel() / C;
    need_cuda(x_);
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = x_.contiguous();
    const int code = dtype_code(x);
    Tensor out = at::empty({C}, x.options().dtype(bf16 ? at::kBFloat16 : at::kFloat));
    const size_t bytes = o1d_colsum_workspace_bytes(rows, (int)C, code);
    Tensor ws = at::empty({(int64_t)std::max<size_t>(bytes, 4)}, x.options().dtype(at::kByte));
    check(o1d_colsum(ptr(x), (float *)out.data_ptr(), ws.data_ptr(), bytes, rows, (int)C, code | (bf16 ? O1D_FLAG_PARAMS_BF16 : 0), stream()),
          "o1d_colsum");
    return out;
}

Tensor pointwise_in(const Tensor &x_, const Tensor &w, const OptTensor &bias) {
    if (x_.dim() != 4) throw py::value_error("expected a 4-D tensor");
    if (w.dim() == 0) throw py::value_error("weight must be [Cout, Cin]");
    need_numel(w, w.size(0) * x_.size(1), "weight");
    if (bias) need_numel(*bias, w.size(0), "bias");
    need_cuda(x_); need_cuda(w); need_cuda(bias);
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = x_.contiguous();
    const int code = dtype_code(x);
    Params p(w, bias);
    Tensor y = at::empty({x.size(0), x.size(2), x.size(3), w.size(0)}, x.options());
    void *st = stream();
    call(p, "o1d_pointwise_in", [&](int pf) {
        return o1d_pointwise_in(ptr(x), (const float *)ptr(p.w), (const float *)ptr(p.b), y.data_ptr(), (int)x.size(0), (int)x.size(1),
                                x.size(2) * x.size(3), (int)w.size(0), code | pf, st);
    });
    return y;
}

// The operator's autograd node (reference: models/dwoconv1d/dwoconv1d.py:18-69), free of Python on the
// backward thread.  An NCHW tensor whose NHWC form has a fast path (`via`) is converted on the way in and
// out, and its NHWC form is what backward keeps.
struct ConvFn : torch::autograd::Function<ConvFn> {
    static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &x_, const Tensor &w, const Tensor &theta,
                          const OptTensor &bias, const Tensor &host, const Tensor &dev, int64_t plan_c, int64_t K, int64_t stride, bool nhwc,
                          bool via, bool identity, bool gelu) {
        (void)theta;
        const Tensor x = via ? transpose(x_, true) : x_.contiguous();
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({x, w});
        ctx->saved_data["host"] = host;
        ctx->saved_data["dev"] = dev;
        ctx->saved_data["p"] = std::vector<int64_t>{plan_c, K, stride, nhwc, via, identity, gelu, bias.has_value()};
        const Tensor y = fprop(x, w, bias, plan_c, K, (int64_t)host.const_data_ptr(), (int64_t)dev.const_data_ptr(), stride, nhwc || via,
                               identity, gelu);
        return via ? transpose(y, false) : y;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        torch::autograd::variable_list out(13);
        Tensor dy = grads[0];
        if (!dy.defined()) return out;
        const auto saved = ctx->get_saved_variables();
        const Tensor &x = saved[0], &w = saved[1];
        const auto p = ctx->saved_data["p"].toIntVector();
        const int64_t plan_c = p[0], K = p[1], stride = p[2], host = (int64_t)ctx->saved_data["host"].toTensor().const_data_ptr(),
                      dev = (int64_t)ctx->saved_data["dev"].toTensor().const_data_ptr();
        const bool nhwc = p[3] || p[4], via = p[4], identity = p[5], gelu = p[6], has_bias = p[7];
        if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
        dy = via ? transpose(dy, true) : dy.contiguous();
        if (ctx->needs_input_grad(0)) {
            out[0] = dgrad(dy, w, plan_c, K, host, dev, x.size(nhwc ? 1 : 2), x.size(nhwc ? 2 : 3), stride, nhwc, identity,
                           gelu ? OptTensor(x) : std::nullopt);
            if (via) out[0] = transpose(out[0], false);
        }
        const bool need_w = ctx->needs_input_grad(1), need_b = has_bias && ctx->needs_input_grad(3);
        if (need_w || need_b) {
            auto [dw, db] = wgrad(dy, x, plan_c, K, host, dev, stride, nhwc, need_b, gelu, is_bf16(w));
            const auto dt = w.scalar_type();             // the bias shares the weight's dtype
            if (need_w) out[1] = dw.scalar_type() == dt ? dw : dw.to(dt);
            if (need_b) out[3] = db->scalar_type() == dt ? *db : db->to(dt);
        }
        return out;
    }
};

// Channels-last LayerNorm (and GELU) with this library's kernels on both passes.
struct LayerNormFn : torch::autograd::Function<LayerNormFn> {
    static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &x_, const Tensor &g, const Tensor &b, double eps, bool gelu) {
        const Tensor x = x_.contiguous();
        ctx->save_for_backward({x, g, b});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["gelu"] = gelu;
        return layer_norm_cl(x, g, b, eps, gelu);
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        auto [dx, dg, db] = layer_norm_cl_bwd(saved[0], grads[0], saved[1], ctx->saved_data["eps"].toDouble(), saved[2],
                                              ctx->saved_data["gelu"].toBool(), true);
        return {ctx->needs_input_grad(0) ? dx : Tensor(), ctx->needs_input_grad(1) ? dg : Tensor(), ctx->needs_input_grad(2) ? db : Tensor(),
                Tensor(), Tensor()};
    }
};
Tensor layer_norm_train(const Tensor &x, const Tensor &g, const Tensor &b, double eps, bool gelu) { return LayerNormFn::apply(x, g, b, eps, gelu); }

// Linear on channels-last activations whose bias gradient is this library's column sum; the two matrix
// products stay with the GEMM library.
struct LinearFn : torch::autograd::Function<LinearFn> {
    static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &x, const Tensor &w, const Tensor &b) {
        ctx->save_for_backward({x, w});
        ctx->saved_data["bias"] = (int64_t)b.scalar_type();
        return at::linear(x, w, b);
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &x = saved[0], &w = saved[1], dy = grads[0].reshape({-1, grads[0].size(-1)});
        torch::autograd::variable_list out(3);
        if (ctx->needs_input_grad(0)) out[0] = dy.matmul(w).reshape(x.sizes());
        if (ctx->needs_input_grad(1)) out[1] = dy.t().matmul(x.reshape({-1, x.size(-1)}));
        if (ctx->needs_input_grad(2)) {
            const auto dt = (at::ScalarType)ctx->saved_data["bias"].toInt();
            out[2] = colsum(dy, dt == at::kBFloat16);
            if (out[2].scalar_type() != dt) out[2] = out[2].to(dt);
        }
        return out;
    }
};
Tensor linear_train(const Tensor &x, const Tensor &w, const Tensor &b) { return LinearFn::apply(x, w, b); }

Tensor conv(const Tensor &x, const Tensor &w, const Tensor &theta, const OptTensor &bias, const Tensor &host, const Tensor &dev,
            int64_t plan_c, int64_t K, int64_t stride, bool nhwc, bool via, bool identity, bool gelu) {
    return ConvFn::apply(x, w, theta, bias, host, dev, plan_c, K, stride, nhwc, via, identity, gelu);
}

}  // namespace

PYBIND11_MODULE(_o1d_torch, m) {
    m.def("set_check", [](py::object f) { g_check = new py::object(std::move(f)); });
    m.def("fprop", &fprop, py::call_guard<py::gil_scoped_release>());
    m.def("dgrad", &dgrad, py::call_guard<py::gil_scoped_release>());
    m.def("wgrad", &wgrad, py::call_guard<py::gil_scoped_release>());
    m.def("conv", &conv, py::call_guard<py::gil_scoped_release>());
    m.def("layer_norm_train", &layer_norm_train, py::call_guard<py::gil_scoped_release>());
    m.def("linear_train", &linear_train, py::call_guard<py::gil_scoped_release>());
    m.def("transpose", &transpose, py::call_guard<py::gil_scoped_release>());
    m.def("layer_norm_cl", &layer_norm_cl, py::call_guard<py::gil_scoped_release>());
    m.def("layer_norm_cl_bwd", &layer_norm_cl_bwd, py::call_guard<py::gil_scoped_release>());
    m.def("colsum", &colsum, py::call_guard<py::gil_scoped_release>());
    m.def("pointwise_in", &pointwise_in, py::call_guard<py::gil_scoped_release>());
}
