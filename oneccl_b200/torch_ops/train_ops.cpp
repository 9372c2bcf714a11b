// Mean softmax cross-entropy whose logits become their own gradient (kernels: csrc/gpu/train_kernels.cu).
#include "torch_ops.hpp"

#include <torch/csrc/autograd/functions/utils.h>

namespace cclx_ops {
namespace {

using torch::autograd::variable_list;

struct SoftmaxXentBackward : torch::autograd::Node {
    Tensor grad; // the logits' memory, which holds their gradient
    int64_t version = 0; // of the logits: the kernel's write is not counted, any later one is
    bool scale = false;

    std::string name() const override {
        return "SoftmaxXentBackward";
    }
    void release_variables() override {
        std::lock_guard<std::mutex> g(mutex_);
        grad.reset();
    }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> g(mutex_);
        if (!grads[0].defined())
            return { Tensor() };
        TORCH_CHECK(grad.defined(), "the logits' gradient has been freed: backward ran through the graph a second time");
        TORCH_CHECK((int64_t)grad._version() == version,
                    "one of the variables needed for gradient computation has been modified by an inplace operation: the logits hold "
                    "their gradient after the fused cross-entropy");
        // the stored gradient assumes d(loss) = 1; scale only when the caller scaled the loss
        return { scale ? grad * grads[0].to(grad.scalar_type()) : grad };
    }
};

Tensor softmax_xent(const Tensor& logits, const Tensor& targets_, int64_t vocab, bool scale) {
    TORCH_CHECK(logits.is_cuda() && targets_.is_cuda(), "the fused cross-entropy takes CUDA tensors");
    no_tangent("the fused cross-entropy", { logits });
    pybind11::gil_scoped_release nogil;
    const Tensor targets = targets_.is_contiguous() ? targets_ : targets_.contiguous();
    const int64_t rows = logits.size(0), cols = logits.size(1);
    Tensor mean;
    if (rows == 0) // the mean of nothing
        mean = at::full({}, std::numeric_limits<float>::quiet_NaN(), logits.options().dtype(at::kFloat).requires_grad(false));
    else {
        void* st = stream_of(logits);
        const Tensor losses = empty_on(logits, { rows }, at::kFloat);
        mean = empty_on(logits, {}, at::kFloat);
        // autograd is not told about the in-place write: the producer of `logits` (a matmul) does not need its output
        // for its own backward
        check(cclx_softmax_xent_mean(logits.data_ptr(), reinterpret_cast<const long long*>(targets.data_ptr<int64_t>()),
                                     losses.data_ptr<float>(), mean.data_ptr<float>(), rows, (int)vocab, logits.stride(0),
                                     1.0f / (float)rows, (int)(cols - vocab), st));
        launches += 2;
    }
    if (torch::autograd::compute_requires_grad(logits)) {
        std::shared_ptr<SoftmaxXentBackward> node(new SoftmaxXentBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(logits));
        node->grad = logits.detach();
        node->version = (int64_t)logits._version();
        node->scale = scale;
        torch::autograd::set_history(mean, node);
    }
    return mean;
}

// one step of the flat AdamW: clipping norm (max_norm > 0) and update
void adamw_step(const Tensor& master, const Tensor& grad, const Tensor& m, const Tensor& v, const std::optional<Tensor>& model,
                int64_t n_decay, double lr, double beta1, double beta2, double eps, double weight_decay, int64_t step,
                double grad_scale, double max_norm, const Tensor& norm, const Tensor& counter, const std::optional<Tensor>& step_dev) {
    pybind11::gil_scoped_release nogil;
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
