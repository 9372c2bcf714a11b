// LayerNorm with the residual addition as an autograd function (kernels: csrc/gpu/nn_kernels.cu).
#include "torch_ops.hpp"

namespace cclx_ops {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// [rows, D] form of a tensor whose last dimension is D
Tensor rows_of(const Tensor& t, int64_t D) {
    Tensor r = t.dim() == 2 ? t : t.reshape({ -1, D });
    return r.is_contiguous() ? r : r.contiguous();
}

Tensor shaped(const Tensor& t, at::IntArrayRef shape) {
    return shape.size() == 2 ? t : t.view(shape);
}

struct AddLayerNorm : torch::autograd::Function<AddLayerNorm> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& res, const Tensor& weight,
                                 const Tensor& bias, double eps) {
        const int64_t D = x.size(-1);
        const Tensor x2 = rows_of(x, D);
        const int64_t rows = x2.size(0);
        void* st = stream_of(x2);
        const Tensor y = empty_on(x2, x2.sizes(), at::kBFloat16);
        const Tensor stats = empty_on(x2, { 2, rows }, at::kFloat); // mean, 1 / standard deviation
        float* mean = stats.data_ptr<float>();
        Tensor total = x2;
        if (res) {
            const Tensor r2 = rows_of(*res, D);
            total = empty_on(x2, x2.sizes(), at::kBFloat16);
            check(cclx_layer_norm_fwd(x2.data_ptr(), r2.data_ptr(), weight.data_ptr(), bias.data_ptr(), y.data_ptr(),
                                      total.data_ptr(), mean, mean + rows, rows, (int)D, (float)eps, st));
        }
        else
            check(cclx_layer_norm_fwd(x2.data_ptr(), nullptr, weight.data_ptr(), bias.data_ptr(), y.data_ptr(), nullptr,
                                      mean, mean + rows, rows, (int)D, (float)eps, st));
        launches += 1;
        ctx->save_for_backward({ total, weight, stats });
        ctx->set_materialize_grads(false); // an unused output costs no zero tensor
        if (res)
            return { shaped(y, x.sizes()), shaped(total, x.sizes()) };
        return { shaped(y, x.sizes()) };
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &total = saved[0], &weight = saved[1], &stats = saved[2];
        const int64_t rows = total.size(0), D = total.size(1);
        const bool has_res = grads.size() == 2; // as many as forward had outputs
        Tensor dsum = has_res ? grads[1] : Tensor();
        if (!grads[0].defined() && !dsum.defined())
            return variable_list(5);
        const Tensor dy = grads[0].defined() ? rows_of(grads[0], D) : at::zeros_like(total);
        if (dsum.defined())
            dsum = rows_of(dsum, D);
        void* st = stream_of(total);
        const Tensor dx = empty_on(total, total.sizes(), at::kBFloat16);
        const Tensor dgamma = empty_on(total, weight.sizes(), at::kBFloat16), dbeta = empty_on(total, weight.sizes(), at::kBFloat16);
        if (rows == 0) {
            dgamma.zero_();
            dbeta.zero_();
        }
        const Tensor ws = empty_on(total, { (int64_t)cclx_layer_norm_bwd_blocks(rows) * 2 * D }, at::kFloat);
        const float* mean = stats.data_ptr<float>();
        check(cclx_layer_norm_bwd_sums(dy.data_ptr(), total.data_ptr(), weight.data_ptr(), mean, mean + rows,
                                       dsum.defined() ? dsum.data_ptr() : nullptr, dx.data_ptr(), dgamma.data_ptr(),
                                       dbeta.data_ptr(), nullptr, 0, ws.data_ptr<float>(), rows, (int)D, st));
        launches += 2;
        const auto shape = grads[0].defined() ? grads[0].sizes() : grads[1].sizes();
        const Tensor d = shaped(dx, shape);
        return { d, has_res ? d : Tensor(), dgamma, dbeta, Tensor() };
    }
};

bool ln_param_ok(const Tensor& p, int64_t D) {
    return p.scalar_type() == at::kBFloat16 && p.is_cuda() && p.numel() == D && p.is_contiguous() && aligned16(p);
}

// whether the fused kernels take this call: bf16 on a GPU, rows of whole 16-byte packs up to 2048 columns
bool layer_norm_ok(const Tensor& x, const std::optional<Tensor>& res, const Tensor& w, const Tensor& b) {
    if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() < 1)
        return false;
    const int64_t D = x.size(-1);
    return D % 8 == 0 && D >= 256 && D <= 2048 && (!x.is_contiguous() || aligned16(x)) &&
           (!res || (res->scalar_type() == at::kBFloat16 && res->sizes() == x.sizes() && (!res->is_contiguous() || aligned16(*res)))) &&
           ln_param_ok(w, D) && ln_param_ok(b, D);
}

// (LayerNorm(x + res), x + res), or None where the kernels do not take the call
pybind11::object add_layer_norm(const Tensor& x, const std::optional<Tensor>& res, const Tensor& w, const Tensor& b, double eps) {
    if (!layer_norm_ok(x, res, w, b))
        return pybind11::none();
    variable_list out;
    {
        pybind11::gil_scoped_release nogil;
        out = AddLayerNorm::apply(x, res, w, b, eps);
    }
    if (res)
        return pybind11::make_tuple(out[0], out[1]);
    return pybind11::cast(out[0]);
}

} // namespace

void bind_nn(pybind11::module_& m) {
    m.def("add_layer_norm", &add_layer_norm);
}

} // namespace cclx_ops
