// Layers of the decoder models as autograd functions (kernels: csrc/gpu/nn_kernels.cu, embedding_kernels.cu).
//
// Bias gradients are column sums of the gradient of a linear layer's output.  The kernel that produces that gradient sums
// it on the way: LayerNorm's backward for the layer in front of a residual addition, GELU's for the first MLP layer, the
// packing of the QKV gradient for the attention projection.  Such an operator takes the bias as an input whose value it
// does not need and returns its gradient; `linear` is then called with defer_bias.
#include "torch_ops.hpp"

#include <ATen/autocast_mode.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

namespace cclx_ops {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// [rows, D] form of a tensor whose last dimension is D
Tensor rows_of(const Tensor& t, int64_t D) {
    Tensor r = t.dim() == 2 ? t : t.reshape({ -1, D });
    r = r.is_contiguous() ? r : r.contiguous();
    return aligned16(r) ? r : r.clone();
}

// the same elements contiguous and 16-byte aligned
Tensor dense(const Tensor& t) {
    const Tensor r = t.is_contiguous() ? t : t.contiguous();
    return aligned16(r) ? r : r.clone();
}

Tensor shaped(const Tensor& t, at::IntArrayRef shape) {
    return shape.size() == 2 ? t : t.view(shape);
}

// the sinks of an operator's parameters, kept with its autograd node
struct Sinks : torch::CustomClassHolder {
    std::vector<SinkRef> s;
};

void keep_sinks(AutogradContext* ctx, std::vector<SinkRef> s) {
    for (const auto& x : s)
        if (x) {
            auto h = c10::make_intrusive<Sinks>();
            h->s = std::move(s);
            ctx->saved_data["sinks"] = c10::IValue::make_capsule(std::move(h));
            return;
        }
}

// Destination of a parameter's gradient: the sink's buffer, or a tensor to return to autograd.
struct ParamGrad {
    SinkRef sink;
    Tensor out;
    bool add = false;

    // `beside`: it will be written on the sink's stream of gradients, not on the current stream.
    // `room`: where the gradient goes if there is no sink (allocated if undefined)
    ParamGrad(const SinkRef& s, const Tensor& like, at::IntArrayRef shape, bool beside = false, Tensor room = Tensor()) : sink(s) {
        if (s) {
            out = s->grad;
            add = beside && s->on_side ? s->take() : s->add();
            s->on_side = beside;
        }
        else
            out = room.defined() ? std::move(room) : empty_on(like, shape, at::kBFloat16);
    }
    void* ptr() const {
        return out.data_ptr();
    }
    void nothing() const { // no row contributes
        if (!add)
            out.zero_();
    }
    Tensor result() const {
        return sink ? Tensor() : out;
    }
    void done() const {
        if (sink)
            sink->report();
    }
};

// Runs `f(defer)`, which launches a kernel that leaves partial sums in `ws` and adds them up unless it can leave their number
// in *defer; then they are added up beside the rest of backward.
template <class F>
void with_sums(const GradStreamRef& beside, const Tensor& ws, int cols, std::initializer_list<const ParamGrad*> outs, F&& f) {
    int n = 0;
    f(beside ? &n : nullptr);
    launches += 2;
    if (!beside || n == 0)
        return;
    void* o[3] = {};
    int k = 0, add = 0;
    for (const ParamGrad* p : outs) {
        add |= (p->add ? 1 : 0) << k;
        o[k++] = p->ptr();
    }
    at::cuda::CUDAEvent ready;
    ready.record(at::cuda::getCurrentCUDAStream(ws.get_device()));
    beside->launch(
        ready, [&] { check(cclx_partial_sums(ws.data_ptr<float>(), n, cols, k, o[0], o[1], o[2], add, stream_of(ws))); }, ws, ws);
}

// the stream of gradients that all of these sinks allow, or none
GradStreamRef beside_of(std::initializer_list<SinkRef> sinks) {
    GradStreamRef b;
    for (const SinkRef& s : sinks) {
        if (!s || !s->beside || (b && b != s->beside))
            return nullptr;
        b = s->beside;
    }
    return b;
}

std::vector<SinkRef> sinks_of(AutogradContext* ctx, size_t n) {
    auto it = ctx->saved_data.find("sinks");
    if (it == ctx->saved_data.end())
        return std::vector<SinkRef>(n);
    return c10::static_intrusive_pointer_cast<Sinks>(it->second.toCapsule())->s;
}

// Written as a plain autograd node: the wrapper of torch::autograd::Function costs several microseconds each way.
struct AddLayerNormBackward : torch::autograd::Node {
    torch::autograd::SavedVariable total, weight;
    Tensor stats; // mean, 1 / standard deviation
    std::vector<SinkRef> sinks;
    bool has_res = false, has_res_bias = false;

    std::string name() const override {
        return "AddLayerNormBackward";
    }
    void release_variables() override {
        std::lock_guard<std::mutex> g(mutex_);
        total.reset_data();
        weight.reset_data();
        stats.reset();
    }
    // gradients of x, the residual, gamma, beta and the bias of the linear layer that produced the residual
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> g(mutex_);
        Tensor dsum = has_res ? grads[1] : Tensor();
        if (!grads[0].defined() && !dsum.defined())
            return variable_list(5);
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor t = total.unpack(shared_from_this()), w = weight.unpack();
        TORCH_CHECK(stats.defined(), "LayerNorm's saved tensors have been freed: backward ran through the graph a second time");
        const auto shape = t.sizes();
        const int64_t D = shape.back(), rows = t.numel() / std::max<int64_t>(D, 1);
        const Tensor dy = grads[0].defined() ? dense(grads[0]) : at::zeros_like(t);
        if (dsum.defined())
            dsum = dense(dsum);
        void* st = stream_of(t);
        const Tensor dx = empty_on(t, shape, at::kBFloat16);
        const int64_t wide[] = { D };
        const bool own = !sinks[0] && !sinks[1];
        const GradStreamRef beside = has_res_bias ? beside_of({ sinks[0], sinks[1], sinks[2] }) : beside_of({ sinks[0], sinks[1] });
        const Tensor both = own ? empty_on(t, { 2 * D }, at::kBFloat16) : Tensor(); // gamma's and beta's gradients are born together
        const ParamGrad dg(sinks[0], t, wide, (bool)beside, own ? part_of(both, 0, wide, at::kBFloat16) : Tensor());
        const ParamGrad db(sinks[1], t, wide, (bool)beside, own ? part_of(both, 2 * D, wide, at::kBFloat16) : Tensor());
        std::optional<ParamGrad> dr;
        if (has_res_bias)
            dr.emplace(sinks[2], t, wide, (bool)beside);
        if (rows == 0) {
            dg.nothing();
            db.nothing();
            if (dr)
                dr->nothing();
        }
        const Tensor ws = empty_on(t, { (int64_t)cclx_layer_norm_bwd_blocks(rows) * (dr ? 3 : 2) * D }, at::kFloat);
        const float* mean = stats.data_ptr<float>();
        auto run = [&](int* defer) {
            check(cclx_layer_norm_bwd_sums(dy.data_ptr(), t.data_ptr(), w.data_ptr(), mean, mean + rows,
                                           dsum.defined() ? dsum.data_ptr() : nullptr, dx.data_ptr(), dg.ptr(), db.ptr(),
                                           dr ? dr->ptr() : nullptr,
                                           (dg.add ? 1 : 0) | (db.add ? 2 : 0) | (dr && dr->add ? 4 : 0), ws.data_ptr<float>(), rows,
                                           (int)D, defer, st));
        };
        if (dr)
            with_sums(beside, ws, (int)D, { &dg, &db, &*dr }, run);
        else
            with_sums(beside, ws, (int)D, { &dg, &db }, run);
        dg.done();
        db.done();
        if (dr)
            dr->done();
        return { dx, has_res ? dx : Tensor(), dg.result(), db.result(), dr ? dr->result() : Tensor() };
    }
};

// {LayerNorm(x + res), x + res}; res_bias: bias of the linear layer that produced `res`
variable_list add_layer_norm_fwd(const Tensor& x, const std::optional<Tensor>& res, const Tensor& weight, const Tensor& bias,
                                 double eps, const std::optional<Tensor>& res_bias, std::vector<SinkRef> sinks) {
    const Tensor none;
    const Tensor &r = res ? *res : none, &rb = res_bias ? *res_bias : none;
    no_tangent("the fused LayerNorm", { x, r, weight, bias, rb });
    const bool grad = torch::autograd::compute_requires_grad(x, r, weight, bias, rb);
    Tensor xd, y, total, stats;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        xd = dense(x);
        const int64_t D = xd.size(-1), rows = xd.numel() / D;
        void* st = stream_of(xd);
        y = empty_on(xd, xd.sizes(), at::kBFloat16);
        stats = empty_on(xd, { 2, rows }, at::kFloat);
        float* mean = stats.data_ptr<float>();
        const Tensor rd = res ? dense(r) : none;
        if (res)
            total = empty_on(xd, xd.sizes(), at::kBFloat16);
        check(cclx_layer_norm_fwd(xd.data_ptr(), res ? rd.data_ptr() : nullptr, weight.data_ptr(), bias.data_ptr(), y.data_ptr(),
                                  res ? total.data_ptr() : nullptr, mean, mean + rows, rows, (int)D, (float)eps, st));
        launches += 1;
    }
    if (grad) {
        std::shared_ptr<AddLayerNormBackward> node(new AddLayerNormBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(x, r, weight, bias, rb));
        node->stats = stats;
        node->sinks = std::move(sinks);
        node->has_res = res.has_value();
        node->has_res_bias = res_bias.has_value();
        torch::autograd::set_history(y, node);
        if (res)
            torch::autograd::set_history(total, node);
        node->total = res ? torch::autograd::SavedVariable(total, true) : torch::autograd::SavedVariable(xd, false);
        node->weight = torch::autograd::SavedVariable(weight, false);
    }
    if (res)
        return { y, total };
    return { y };
}

bool bf16_cuda(const Tensor& t) {
    return t.is_cuda() && t.scalar_type() == at::kBFloat16;
}

// whether the kernels can write the gradient of bias `b` of a layer with `n` outputs, beside `x`
bool bias_ok(const Tensor& b, const Tensor& x, int64_t n) {
    return bf16_cuda(b) && b.device() == x.device() && b.dim() == 1 && b.size(0) == n;
}

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

Tensor tensor_of(const pybind11::object& o) {
    return o.cast<Tensor>();
}
std::optional<Tensor> maybe_tensor(const pybind11::object& o) {
    return o.is_none() ? std::optional<Tensor>() : std::optional<Tensor>(o.cast<Tensor>());
}

// (LayerNorm(x + res), x + res), or None where the kernels do not take the call
pybind11::object add_layer_norm(const Tensor& x, const std::optional<Tensor>& res, const pybind11::object& w_,
                                const pybind11::object& b_, double eps, const pybind11::object& res_bias_) {
    const Tensor w = tensor_of(w_), b = tensor_of(b_);
    if (!layer_norm_ok(x, res, w, b))
        return pybind11::none();
    const auto res_bias = maybe_tensor(res_bias_);
    if (res_bias && (!res || !bias_ok(*res_bias, x, x.size(-1))))
        return pybind11::none();
    std::vector<SinkRef> sinks{ sink_of(w_), sink_of(b_), sink_of(res_bias_) };
    variable_list out;
    {
        pybind11::gil_scoped_release nogil;
        out = add_layer_norm_fwd(x, res, w, b, eps, res_bias, std::move(sinks));
    }
    if (res)
        return pybind11::make_tuple(out[0], out[1]);
    return pybind11::cast(out[0]);
}

// bias gradient: column sums of a gradient of [rows, N]
void column_sums(const Tensor& dy, const ParamGrad& out) {
    const int64_t rows = dy.size(0), N = dy.size(1);
    if (rows == 0)
        return out.nothing();
    const Tensor ws = empty_on(dy, { (int64_t)cclx_map_colsum_workspace(rows, (int)N) }, at::kFloat);
    check(cclx_colsum(dy.data_ptr(), out.ptr(), out.add, ws.data_ptr<float>(), rows, (int)N, stream_of(dy)));
    launches += 2;
}

// Gradient of a linear layer's weight: into its sink, if possible beside the rest of backward, or to autograd (`out`).
struct WeightGrad {
    SinkRef sink;
    bool beside;
    at::cuda::CUDAEvent ready; // the gradient of the layer's output is there
    Tensor out;

    WeightGrad(const SinkRef& s, const Tensor& dy) : sink(s), beside(s && s->beside) {
        if (beside)
            ready.record(at::cuda::getCurrentCUDAStream(dy.get_device()));
    }
    void product(const Tensor& dy, const Tensor& x, bool needed) {
        if (!sink) {
            if (needed)
                out = dy.t().mm(x);
            return;
        }
        GradSink& s = *sink;
        const bool add = beside && s.on_side ? s.take() : s.add();
        auto f = [&] {
            if (add)
                s.grad.addmm_(dy.t(), x);
            else
                at::mm_out(s.grad, dy.t(), x);
        };
        if (beside) {
            s.beside->launch(ready, f, dy, x);
            s.on_side = true;
        }
        else
            f();
    }
};

// cuBLAS products with the weight gradient accumulated straight into its sink, if possible beside the rest of backward.
struct Linear : torch::autograd::Function<Linear> {
    // bias_grad: computed here (else another operator returns it); report: this is the weight's last contribution
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias,
                                 bool bias_grad, bool report, std::vector<SinkRef> sinks) {
        const Tensor x2 = x.dim() == 2 ? x : x.reshape({ -1, x.size(-1) });
        ctx->save_for_backward({ x2, weight });
        ctx->saved_data["flags"] = (int64_t)((bias && bias_grad ? 1 : 0) | (report ? 2 : 0));
        ctx->saved_data["shape"] = x.sizes().vec();
        keep_sinks(ctx, std::move(sinks));
        const Tensor y = bias ? at::addmm(*bias, x2, weight.t()) : x2.mm(weight.t());
        if (x.dim() == 2)
            return { y };
        auto shape = x.sizes().vec();
        shape.back() = weight.size(0);
        return { y.view(shape) };
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &x2 = saved[0], &weight = saved[1];
        const auto sinks = sinks_of(ctx, 2);
        const int64_t flags = ctx->saved_data["flags"].toInt();
        const Tensor dy = rows_of(grads[0], grads[0].size(-1));
        Tensor dx, db;
        WeightGrad dw(sinks[0], dy);
        if (ctx->needs_input_grad(0))
            dx = dy.mm(weight).view(ctx->saved_data["shape"].toIntVector());
        dw.product(dy, x2, ctx->needs_input_grad(1));
        if (flags & 1) {
            const ParamGrad g(sinks[1], dy, { dy.size(1) });
            column_sums(dy, g);
            db = g.result();
            g.done();
        }
        if (sinks[0] && flags & 2)
            sinks[0]->report();
        return { dx, dw.out, db, Tensor(), Tensor(), Tensor() };
    }
};

// None where the operator does not take the call
pybind11::object linear(const Tensor& x, const pybind11::object& w_, const pybind11::object& b_, bool bias_grad, bool report) {
    const Tensor w = tensor_of(w_);
    const auto b = maybe_tensor(b_);
    if (!bf16_cuda(x) || !bf16_cuda(w) || w.dim() != 2 || w.size(0) % 8 != 0 || (b && !bias_ok(*b, x, w.size(0))))
        return pybind11::none();
    std::vector<SinkRef> sinks{ sink_of(w_), sink_of(b_) };
    pybind11::gil_scoped_release nogil;
    Tensor y = Linear::apply(x, w, b, bias_grad, report, std::move(sinks))[0];
    pybind11::gil_scoped_acquire gil;
    return pybind11::cast(y);
}

// tanh-form GELU of a linear layer's output u = ... + bias; backward also returns the bias gradient
struct BiasGelu : torch::autograd::Function<BiasGelu> {
    static variable_list forward(AutogradContext* ctx, const Tensor& u, const Tensor& bias, std::vector<SinkRef> sinks) {
        const Tensor u2 = rows_of(u, u.size(-1));
        const Tensor y = empty_on(u2, u2.sizes(), at::kBFloat16);
        check(cclx_gelu_fwd(u2.data_ptr(), y.data_ptr(), u2.numel(), stream_of(u2)));
        launches += 1;
        ctx->save_for_backward({ u2, bias });
        keep_sinks(ctx, std::move(sinks));
        return { shaped(y, u.sizes()) };
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor& u = saved[0];
        const int64_t rows = u.size(0), N = u.size(1);
        const Tensor dy = rows_of(grads[0], N), du = empty_on(u, u.sizes(), at::kBFloat16);
        const SinkRef sink = sinks_of(ctx, 1)[0];
        const GradStreamRef beside = beside_of({ sink });
        const ParamGrad g(sink, u, saved[1].sizes(), (bool)beside);
        if (rows == 0)
            g.nothing();
        const Tensor ws = empty_on(u, { (int64_t)cclx_map_colsum_workspace(rows, (int)N) }, at::kFloat);
        with_sums(beside, ws, (int)N, { &g }, [&](int* defer) {
            check(cclx_gelu_bwd_colsum(dy.data_ptr(), u.data_ptr(), du.data_ptr(), g.ptr(), g.add, ws.data_ptr<float>(), rows, (int)N,
                                       defer, stream_of(u)));
        });
        g.done();
        return { shaped(du, grads[0].sizes()), g.result(), Tensor() };
    }
};

// None where the operator does not take the call
pybind11::object bias_gelu(const Tensor& u, const pybind11::object& b_) {
    const Tensor b = tensor_of(b_);
    if (!bf16_cuda(u) || u.dim() < 1 || u.size(-1) == 0 || u.size(-1) % 8 != 0 || !bias_ok(b, u, u.size(-1)))
        return pybind11::none();
    std::vector<SinkRef> sinks{ sink_of(b_) };
    pybind11::gil_scoped_release nogil;
    Tensor y = BiasGelu::apply(u, b, std::move(sinks))[0];
    pybind11::gil_scoped_acquire gil;
    return pybind11::cast(y);
}

// gelu(x W1^T + b1) W2^T + b2 with the GELU and its gradient inside the products (csrc/gpu/gemm_mlp.cu).  b2's gradient is left to
// the operator that consumes the output.
struct Mlp : torch::autograd::Function<Mlp> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const Tensor& b1, const Tensor& w2,
                                 const Tensor& b2, std::vector<SinkRef> sinks) {
        const int64_t D = x.size(-1), N = w1.size(0);
        const Tensor x2 = rows_of(x, D), w = dense(w1), b = dense(b1);
        const Tensor u = empty_on(x2, { x2.size(0), N }, at::kBFloat16), g = empty_on(x2, { x2.size(0), N }, at::kBFloat16);
        check(cclx_linear_gelu(x2.data_ptr(), w.data_ptr(), b.data_ptr(), u.data_ptr(), g.data_ptr(), (int)x2.size(0), (int)N, (int)D,
                               stream_of(x2)));
        launches += 1;
        ctx->save_for_backward({ x2, w1, b1, w2, u, g });
        ctx->saved_data["shape"] = x.sizes().vec();
        keep_sinks(ctx, std::move(sinks));
        const Tensor y = at::addmm(b2, g, w2.t());
        auto shape = x.sizes().vec();
        shape.back() = w2.size(0);
        return { y.view(shape) };
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &x2 = saved[0], &w1 = saved[1], &w2 = saved[3], &u = saved[4], &g = saved[5];
        const auto sinks = sinks_of(ctx, 3); // of w1, b1, w2
        const int64_t rows = u.size(0), N = u.size(1), K = w2.size(0);
        const Tensor dy = rows_of(grads[0], K), w = dense(w2);
        WeightGrad d2(sinks[2], dy);
        const Tensor du = empty_on(u, u.sizes(), at::kBFloat16);
        const GradStreamRef beside = beside_of({ sinks[1] });
        const ParamGrad db(sinks[1], u, saved[2].sizes(), (bool)beside);
        const int n = cclx_linear_gelu_bwd_rows((int)rows);
        const Tensor ws = empty_on(u, { n * N }, at::kFloat);
        void* st = stream_of(u);
        with_sums(beside, ws, (int)N, { &db }, [&](int* defer) {
            check(cclx_linear_gelu_bwd(dy.data_ptr(), w.data_ptr(), u.data_ptr(), du.data_ptr(), ws.data_ptr<float>(), (int)rows, (int)N,
                                       (int)K, st));
            if (defer)
                *defer = n;
            else
                check(cclx_partial_sums(ws.data_ptr<float>(), n, (int)N, 1, db.ptr(), nullptr, nullptr, db.add, st));
        });
        d2.product(dy, g, ctx->needs_input_grad(3));
        // in the order of the operators of their own: ranks with batches of different sizes reduce their buckets in the same order
        if (sinks[2])
            sinks[2]->report();
        db.done();
        WeightGrad d1(sinks[0], du);
        Tensor dx;
        if (ctx->needs_input_grad(0))
            dx = du.mm(w1).view(ctx->saved_data["shape"].toIntVector());
        d1.product(du, x2, ctx->needs_input_grad(1));
        if (sinks[0])
            sinks[0]->report();
        return { dx, d1.out, db.result(), d2.out, Tensor(), Tensor() };
    }
};

// None where the operator does not take the call, and with `if_faster` where products of their own are expected to be faster
pybind11::object mlp(const Tensor& x, const pybind11::object& w1_, const pybind11::object& b1_, const pybind11::object& w2_,
                     const pybind11::object& b2_, bool if_faster) {
    const Tensor w1 = tensor_of(w1_), b1 = tensor_of(b1_), w2 = tensor_of(w2_), b2 = tensor_of(b2_);
    if (!bf16_cuda(x) || x.dim() < 1 || !bf16_cuda(w1) || !bf16_cuda(w2) || w1.dim() != 2 || w2.dim() != 2 ||
        w1.device() != x.device() || w2.device() != x.device() || w1.size(1) != x.size(-1) || w2.size(1) != w1.size(0) ||
        w1.size(0) % 8 != 0 || w1.size(1) % 8 != 0 || w2.size(0) % 8 != 0 || x.numel() == 0 || w1.numel() == 0 || w2.numel() == 0 ||
        !bias_ok(b1, x, w1.size(0)) || !bias_ok(b2, x, w2.size(0)))
        return pybind11::none();
    // autocast to another type gives the second product, and so its gradient, that type
    if (at::autocast::is_autocast_enabled(at::kCUDA) && at::autocast::get_autocast_dtype(at::kCUDA) != at::kBFloat16)
        return pybind11::none();
    const int64_t rows = x.numel() / x.size(-1);
    if (rows * std::max(w1.size(0), w2.size(0)) >= (int64_t)1 << 31)
        return pybind11::none();
    set_device(x.get_device()); // whose SMs are counted
    int answer = 0;
    check(cclx_mlp_preferred((int)rows, (int)w1.size(0), &answer));
    if (answer < (if_faster ? 2 : 1))
        return pybind11::none();
    std::vector<SinkRef> sinks{ sink_of(w1_), sink_of(b1_), sink_of(w2_) };
    pybind11::gil_scoped_release nogil;
    Tensor y = Mlp::apply(x, w1, b1, w2, b2, std::move(sinks))[0];
    pybind11::gil_scoped_acquire gil;
    return pybind11::cast(y);
}

// views of a packed QKV projection for the attention call; backward assembles the packed gradient in one pass that also
// sums the bias gradient
struct SplitQKV : torch::autograd::Function<SplitQKV> {
    static variable_list forward(AutogradContext* ctx, const Tensor& qkv, const std::optional<Tensor>& bias, int64_t n_head,
                                 std::vector<SinkRef> sinks) {
        const int64_t B = qkv.size(0), S = qkv.size(1), D = qkv.size(2) / 3, dh = D / n_head;
        const Tensor parts = qkv.view({ B, S, 3, n_head, dh }).permute({ 2, 0, 3, 1, 4 }); // [3, B, H, S, dh] views
        ctx->saved_data["heads"] = n_head;
        ctx->saved_data["bias"] = bias.has_value();
        keep_sinks(ctx, std::move(sinks));
        return { parts[0], parts[1], parts[2] };
    }

    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const bool bias = ctx->saved_data["bias"].toBool();
        const int64_t B = g[0].size(0), H = g[0].size(1), S = g[0].size(2), dh = g[0].size(3), N = 3 * H * dh;
        const Tensor out = empty_on(g[0], { B, S, N }, at::kBFloat16);
        const void* src[3];
        long long strides[9];
        for (int p = 0; p < 3; p++) { // gradients are indexed [B, H, S, dh]
            if (g[p].scalar_type() != at::kBFloat16 || g[p].stride(3) != 1 || g[p].stride(0) % 8 || g[p].stride(1) % 8 ||
                g[p].stride(2) % 8 || !aligned16(g[p]))
                g[p] = g[p].to(at::kBFloat16).contiguous().clone();
            src[p] = g[p].data_ptr();
            strides[3 * p] = g[p].stride(0);
            strides[3 * p + 1] = g[p].stride(2);
            strides[3 * p + 2] = g[p].stride(1);
        }
        // without a bias the sums go nowhere
        const SinkRef sink = sinks_of(ctx, 1)[0];
        const GradStreamRef beside = beside_of({ sink });
        const ParamGrad db(sink, out, { N }, (bool)beside);
        if (B * S == 0)
            db.nothing();
        const Tensor ws = empty_on(out, { (int64_t)cclx_map_colsum_workspace(B * S, (int)N) }, at::kFloat);
        with_sums(beside, ws, (int)N, { &db }, [&](int* defer) {
            check(cclx_qkv_grad_colsum(src, strides, out.data_ptr(), db.ptr(), db.add, ws.data_ptr<float>(), (int)B, (int)S, (int)H,
                                       (int)dh, defer, stream_of(out)));
        });
        db.done();
        return { out, bias ? db.result() : Tensor(), Tensor(), Tensor() };
    }
};

pybind11::object split_qkv(const Tensor& qkv, int64_t n_head, const pybind11::object& b_) {
    if (!bf16_cuda(qkv) || qkv.dim() != 3 || !qkv.is_contiguous() || qkv.size(2) / 3 / n_head % 8 != 0)
        return pybind11::none();
    const auto b = maybe_tensor(b_);
    if (b && !bias_ok(*b, qkv, qkv.size(2)))
        return pybind11::none();
    std::vector<SinkRef> sinks{ sink_of(b_) };
    variable_list out;
    {
        pybind11::gil_scoped_release nogil;
        out = SplitQKV::apply(qkv, b, n_head, std::move(sinks));
    }
    return pybind11::make_tuple(out[0], out[1], out[2]);
}

// An id outside the table is found by the kernel: its row is NaN, and the next call on any thread reports it.
void embed_check() {
    TORCH_CHECK_INDEX(!cclx_embed_bad_id(), "an earlier embedding was given a token id outside its table");
}

// token embedding + position embedding of [B, S] ids
struct Embed : torch::autograd::Function<Embed> {
    static variable_list forward(AutogradContext* ctx, const Tensor& idx, const Tensor& tokens, const Tensor& positions,
                                 std::vector<SinkRef> sinks) {
        const int64_t B = idx.size(0), S = idx.size(1), D = tokens.size(1);
        const Tensor out = empty_on(tokens, { B, S, D }, at::kBFloat16);
        check(cclx_embed_fwd(reinterpret_cast<const long long*>(idx.data_ptr<int64_t>()), tokens.data_ptr(), positions.data_ptr(),
                             out.data_ptr(), B * S, (int)S, (int)tokens.size(0), (int)D, stream_of(tokens)));
        launches += 1;
        ctx->save_for_backward({ idx, tokens, positions });
        keep_sinks(ctx, std::move(sinks));
        return { out };
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        embed_check();
        const auto saved = ctx->get_saved_variables();
        const Tensor &idx = saved[0], &tokens = saved[1], &positions = saved[2];
        const int64_t D = tokens.size(1);
        const Tensor dx = rows_of(grads[0], D);
        const auto sinks = sinks_of(ctx, 2);
        const ParamGrad gt(sinks[0], tokens, tokens.sizes()), gp(sinks[1], positions, positions.sizes());
        if (!gt.add) // only the rows of tokens that occur are touched
            gt.out.zero_();
        const Tensor ws = empty_on(dx, { idx.numel() }, at::kByte);
        check(cclx_embed_bwd(reinterpret_cast<const long long*>(idx.data_ptr<int64_t>()), dx.data_ptr(), gt.ptr(), gp.ptr(), gp.add,
                             (int)idx.size(0), (int)idx.size(1), (int)tokens.size(0), (int)positions.size(0), (int)D,
                             ws.data_ptr(), stream_of(dx)));
        launches += 2;
        gp.done();
        gt.done();
        return { Tensor(), gt.result(), gp.result(), Tensor() };
    }
};

// None where the operator does not take the call
pybind11::object embed(const Tensor& idx_, const pybind11::object& tokens_, const pybind11::object& positions_) {
    const Tensor tokens = tensor_of(tokens_), positions = tensor_of(positions_);
    if (!bf16_cuda(tokens) || !bf16_cuda(positions) || !idx_.is_cuda() || idx_.scalar_type() != at::kLong || idx_.dim() != 2 ||
        idx_.numel() > cclx_embed_bwd_max_ids() || tokens.size(1) % 8 != 0 || positions.size(1) != tokens.size(1) ||
        idx_.size(1) > positions.size(0) || idx_.numel() == 0 || !tokens.is_contiguous() || !positions.is_contiguous() ||
        !aligned16(tokens) || !aligned16(positions))
        return pybind11::none();
    embed_check();
    const Tensor idx = idx_.contiguous();
    std::vector<SinkRef> sinks{ sink_of(tokens_), sink_of(positions_) };
    pybind11::gil_scoped_release nogil;
    const Tensor y = Embed::apply(idx, tokens, positions, std::move(sinks))[0];
    pybind11::gil_scoped_acquire gil;
    return pybind11::cast(y);
}

Tensor colsum(const Tensor& dy) {
    const ParamGrad g(nullptr, dy, { dy.size(1) });
    column_sums(dy, g);
    return g.out;
}

} // namespace

void bind_nn(pybind11::module_& m) {
    m.def("layer_norm_ok", &layer_norm_ok);
    m.def("add_layer_norm", &add_layer_norm, pybind11::arg("x"), pybind11::arg("res"), pybind11::arg("weight"),
          pybind11::arg("bias"), pybind11::arg("eps"), pybind11::arg("res_bias") = pybind11::none());
    m.def("linear", &linear);
    m.def("bias_gelu", &bias_gelu);
    m.def("mlp", &mlp, pybind11::arg("x"), pybind11::arg("w1"), pybind11::arg("b1"), pybind11::arg("w2"), pybind11::arg("b2"),
          pybind11::arg("if_faster") = false);
    m.def("split_qkv", &split_qkv);
    m.def("embed", &embed);
    m.def("embed_check", &embed_check);
    m.def("colsum", &colsum);
}

} // namespace cclx_ops
