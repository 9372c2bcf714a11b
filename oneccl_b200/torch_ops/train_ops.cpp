// Mean softmax cross-entropy whose logits become their own gradient (kernels: csrc/gpu/train_kernels.cu).
#include "torch_ops.hpp"

namespace cclx_ops {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct SoftmaxXent : torch::autograd::Function<SoftmaxXent> {
    static variable_list forward(AutogradContext* ctx, const Tensor& logits, const Tensor& targets, int64_t vocab, bool scale) {
        const int64_t rows = logits.size(0), cols = logits.size(1);
        // autograd is not told about the in-place write: the producer of `logits` (a matmul) does not need its output
        // for its own backward
        ctx->save_for_backward({ logits });
        ctx->saved_data["scale"] = scale;
        if (rows == 0) // the mean of nothing
            return { at::full({}, std::numeric_limits<float>::quiet_NaN(), logits.options().dtype(at::kFloat)) };
        void* st = stream_of(logits);
        const Tensor losses = empty_on(logits, { rows }, at::kFloat), mean = empty_on(logits, {}, at::kFloat);
        check(cclx_softmax_xent_mean(logits.data_ptr(), reinterpret_cast<const long long*>(targets.data_ptr<int64_t>()),
                                     losses.data_ptr<float>(), mean.data_ptr<float>(), rows, (int)vocab, logits.stride(0),
                                     1.0f / (float)rows, (int)(cols - vocab), st));
        launches += 2;
        return { mean };
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        Tensor g = ctx->get_saved_variables()[0];
        // the stored gradient assumes d(loss) = 1; scale only when the caller scaled the loss
        if (grads[0].defined() && ctx->saved_data["scale"].toBool())
            g = g * grads[0].to(g.scalar_type());
        return { g, Tensor(), Tensor(), Tensor() };
    }
};

Tensor softmax_xent(const Tensor& logits, const Tensor& targets, int64_t vocab, bool scale) {
    TORCH_CHECK(logits.is_cuda() && targets.is_cuda(), "the fused cross-entropy takes CUDA tensors");
    const Tensor t = targets.is_contiguous() ? targets : targets.contiguous();
    pybind11::gil_scoped_release nogil;
    return SoftmaxXent::apply(logits, t, vocab, scale)[0];
}

// one step of the flat AdamW: clipping norm (max_norm > 0) and update
void adamw_step(const Tensor& master, const Tensor& grad, const Tensor& m, const Tensor& v, const std::optional<Tensor>& model,
                int64_t n_decay, double lr, double beta1, double beta2, double eps, double weight_decay, int64_t step,
                double grad_scale, double max_norm, const Tensor& norm, const Tensor& counter, const std::optional<Tensor>& step_dev) {
    const int dt = grad.scalar_type() == at::kBFloat16 ? 11 : grad.scalar_type() == at::kFloat ? 9 : -1;
    void* st = stream_of(master);
    const bool clip = max_norm > 0;
    const Tensor scratch =
        clip ? empty_on(master, { (int64_t)cclx_adamw_step_scratch(master.numel(), dt) }, at::kFloat) : Tensor();
    check(cclx_adamw_step(master.data_ptr<float>(), grad.data_ptr(), dt, m.data_ptr<float>(), v.data_ptr<float>(),
                          model ? model->data_ptr() : nullptr, master.numel(), n_decay, (float)lr, (float)beta1, (float)beta2,
                          (float)eps, (float)weight_decay, (int)step, (float)grad_scale, (float)max_norm, norm.data_ptr<float>(),
                          clip ? scratch.data_ptr<float>() : nullptr, reinterpret_cast<unsigned*>(counter.data_ptr<int>()),
                          step_dev ? step_dev->data_ptr<int>() : nullptr, st));
    launches += clip || step_dev ? 2 : 1;
}

} // namespace

void bind_train(pybind11::module_& m) {
    m.def("adamw_step", &adamw_step);
    m.def("softmax_xent", &softmax_xent);
}

} // namespace cclx_ops
