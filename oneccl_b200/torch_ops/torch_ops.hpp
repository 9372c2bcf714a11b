// Shared pieces of the torch-side operators (host code of oneccl_b200.ops in C++): stream and device of a call, error
// translation, the launch counter, prototypes of the kernel entry points in libccl_b200.so.
//
// Why C++: an operator of a small tensor costs more host time than GPU time.  Written as Python autograd functions over
// ctypes, LayerNorm forward + backward took 125 to 190 us of host time around 42 us of kernels.
#pragma once
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>
#include <deque>
#include <functional>
#include <initializer_list>
#include <mutex>
#include <optional>
#include <stdexcept>
#include <string>

extern "C" {
const char* cclx_last_error();
int cclx_set_device(int dev);
int cclx_layer_norm_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* sum_out, float* mean,
                        float* rstd, size_t rows, int D, float eps, void* stream);
int cclx_layer_norm_bwd_blocks(size_t rows);
int cclx_layer_norm_bwd_sums(const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                             const void* dres, void* dx, void* dgamma, void* dbeta, void* dxsum, int add,
                             float* workspace, size_t rows, int D, int* defer, void* stream);
int cclx_dc_allreduce(void* h, const void* const* send, void* const* recv, size_t count, int dt_in, int dt_out, int op, int algo,
                      int blocks, float scale, int do_scale, void* stream);
int cclx_moe_route_one_block();
int cclx_moe_route(const float* logits, int n_tokens, int n_experts, int topk, long long* idx, float* wts, long long* counts,
                   long long* order, long long* pos, void* scratch, void* stream);
int cclx_moe_dispatch(void* h, const void* const* x, const long long* const* order, const long long* const* send_counts,
                      int* const* meta, size_t n_items, int topk, int hidden, const void* recv_buf, size_t cap_rows,
                      const void* cnt_table, int blocks, void* stream);
int cclx_moe_combine_peer(void* h, const long long* const* expert, const long long* const* pos, const float* const* weight,
                          void* const* out, int* const* meta, size_t n_items, int topk, int hidden, const void* expert_out,
                          int blocks, void* stream);
size_t cclx_map_colsum_workspace(size_t rows, int N);
int cclx_colsum(const void* x, void* out, int add, float* workspace, size_t rows, int N, void* stream);
int cclx_gelu_fwd(const void* x, void* y, size_t n, void* stream);
int cclx_gelu_bwd_colsum(const void* dy, const void* x, void* dx, void* colsum, int add, float* workspace, size_t rows, int N,
                         int* defer, void* stream);
int cclx_qkv_grad_colsum(const void* const* src, const long long* strides, void* out, void* colsum, int add, float* workspace,
                         int B, int S, int H, int dh, int* defer, void* stream);
int cclx_partial_sums(const float* workspace, int n, int cols, int outputs, void* out0, void* out1, void* out2, int add, void* stream);
int cclx_embed_fwd(const long long* idx, const void* tokens, const void* positions, void* out, size_t n, int S, int table_rows,
                   int D, void* stream);
int cclx_embed_bad_id();
int cclx_embed_bwd_max_ids();
int cclx_embed_bwd(const long long* idx, const void* dx, void* token_grad, void* pos_grad, int add_pos, int B, int S,
                   int token_rows, int pos_rows, int D, void* workspace, void* stream);
int cclx_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, int ctas, void* err_words,
                   void* stream);
int cclx_gemm_bf16_2sm(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, int clusters,
                       void* err_words, void* stream);
int cclx_gemm_bf16_rows(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, const void* rows_dev,
                        void* err_words, void* stream);
int cclx_mlp_preferred(int M, int N, int* answer);
int cclx_linear_gelu(const void* x, const void* w1, const void* bias, void* u, void* g, int M, int N, int K, void* stream);
int cclx_linear_gelu_bwd_rows(int M);
int cclx_linear_gelu_bwd(const void* dy, const void* w2, const void* u, void* du, float* partial, int M, int N, int K, void* stream);
int cclx_adamw_step(float* master, const void* grad, int grad_dt, float* m, float* v, void* model_bf16, size_t n,
                    size_t n_decay, float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                    float grad_scale, float max_norm, float* sq_norm, float* scratch, unsigned* counter,
                    int* step_dev, void* stream);
size_t cclx_adamw_step_scratch(size_t n, int grad_dt);
int cclx_softmax_xent_mean(void* logits_bf16, const long long* targets, float* loss_rows, float* mean_loss, size_t rows,
                           int vocab, size_t ld, float grad_scale, int pad_cols, void* stream);
}

namespace cclx_ops {

using at::Tensor;

// A contiguous tensor over bytes [offset, ...) of another's storage (offset a multiple of the element size), made without
// the dispatcher: outputs of a small operator that are born together share one allocation.
inline Tensor part_of(const Tensor& base, size_t offset, at::IntArrayRef sizes, at::ScalarType dtype) {
    auto impl = c10::make_intrusive<c10::TensorImpl>(c10::Storage(base.storage()), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                     c10::scalarTypeToTypeMeta(dtype));
    impl->set_storage_offset((int64_t)(offset / c10::elementSize(dtype)));
    impl->set_sizes_contiguous(sizes);
    return Tensor(std::move(impl));
}

// becomes oneccl_b200.CclError in Python
struct ccl_error : std::runtime_error {
    using std::runtime_error::runtime_error;
};

inline void check(int rc) {
    if (rc != 0)
        throw ccl_error(cclx_last_error());
}

// The library has its own CUDA runtime, whose current device is per thread as well: it follows the device of the call
// (autograd runs backward on threads of its own).
inline void set_device(int dev) {
    check(cclx_set_device(dev));
}

inline void* stream_of(const Tensor& t) {
    const int dev = t.get_device();
    set_device(dev);
    return at::cuda::getCurrentCUDAStream(dev).stream();
}

// Operators written as plain autograd nodes have backward alone: a tangent must not get lost in them.
inline void no_tangent(const char* op, std::initializer_list<std::reference_wrapper<const Tensor>> inputs) {
    for (const Tensor& t : inputs)
        TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(0).defined(), "forward-mode differentiation is not implemented for ", op);
}

extern std::atomic<long long> launches; // kernels of the library launched through this module

inline bool aligned16(const Tensor& t) {
    return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}

// an uninitialised contiguous tensor on the device of `like`, without the dispatcher's round trip
inline Tensor empty_on(const Tensor& like, at::IntArrayRef sizes, at::ScalarType dtype) {
    return at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt);
}

// A stream of their own for weight gradients that go to sinks: nothing else in backward waits for them, products of a few
// hundred tokens leave most SMs idle, and a long product's last wave some.  One per DataParallel.
//
// The operands of a product must outlive it, but the allocator knows them as memory of the stream that is current at the launch:
// the operands of the last DEPTH launches are kept, and their stream waits for the oldest before its operands go, whichever
// stream is current by then.  The final sums of bias, gamma and beta gradients run there as well.
class GradStream {
public:
    explicit GradStream(int dev) : stream_(at::cuda::getStreamFromPool(false, (c10::DeviceIndex)dev)) {}

    // runs `product` there once what the current stream has done up to `ready` is done
    template <class F>
    void launch(at::cuda::CUDAEvent& ready, F&& product, const Tensor& a, const Tensor& b) {
        const auto current = at::cuda::getCurrentCUDAStream(a.get_device());
        std::lock_guard<std::mutex> g(mu_);
        ready.block(stream_);
        {
            at::cuda::CUDAStreamGuard guard(stream_);
            product();
        }
        held_.push_back({ {}, a, b, current });
        held_.back().done.record(stream_);
        if (held_.size() > DEPTH) {
            held_.front().done.block(held_.front().home);
            held_.pop_front();
        }
    }
    // `s` waits for everything launched since the last finish()
    void join(at::cuda::CUDAStream s) {
        std::lock_guard<std::mutex> g(mu_);
        if (!held_.empty())
            held_.back().done.block(s);
    }
    // the same for the current stream and those that the operands belong to, at the end of a step
    void finish() {
        std::lock_guard<std::mutex> g(mu_);
        const auto current = at::cuda::getCurrentCUDAStream(stream_.device_index());
        if (!held_.empty())
            held_.back().done.block(current);
        for (size_t i = 0; i < held_.size(); i++)
            if (held_[i].home != current && (i == 0 || held_[i].home != held_[i - 1].home))
                held_.back().done.block(held_[i].home);
        held_.clear();
    }
    uintptr_t handle() const {
        return reinterpret_cast<uintptr_t>(stream_.stream());
    }

private:
    static constexpr size_t DEPTH = 16; // two transformer blocks
    struct entry {
        at::cuda::CUDAEvent done;
        Tensor a, b;
        at::cuda::CUDAStream home;
    };
    at::cuda::CUDAStream stream_;
    std::deque<entry> held_;
    std::mutex mu_;
};
typedef std::shared_ptr<GradStream> GradStreamRef;

// Where a parameter's gradient goes when its layer accumulates it itself: a view of DataParallel's flat gradient.  `fresh`
// says that the buffer still holds the last step's gradient, so that the first contribution overwrites it (a product with
// beta = 0 instead of clearing the buffer and reading it back).  `callback` (no argument) does the bucket accounting;
// it must not keep the parameter alive, which owns this object.
struct GradSink {
    Tensor grad;
    PyObject* callback;
    bool fresh = false;
    GradStreamRef beside; // set during a step that ends by finishing it: weight gradients may run there
    bool on_side = false; // the last contribution did
    static std::atomic<int> live;

    GradSink(Tensor g, pybind11::object cb) : grad(std::move(g)), callback(cb.release().ptr()) {
        live++;
    }
    ~GradSink() {
        live--;
        if (Py_IsInitialized()) {
            pybind11::gil_scoped_acquire gil;
            Py_XDECREF(callback);
        }
    }
    // whether a contribution is added (or overwrites); from then on they are.  The current stream may write afterwards.
    bool add() {
        if (on_side && beside)
            beside->join(at::cuda::getCurrentCUDAStream(grad.get_device()));
        on_side = false;
        return take();
    }
    bool take() {
        const bool a = !fresh;
        fresh = false;
        return a;
    }
    void report() {
        pybind11::gil_scoped_acquire gil;
        pybind11::reinterpret_borrow<pybind11::object>(callback)();
    }
};
typedef std::shared_ptr<GradSink> SinkRef;
SinkRef sink_of(const pybind11::object& param); // null without one

void bind_nn(pybind11::module_& m);
void bind_train(pybind11::module_& m);
void bind_gemm(pybind11::module_& m);
void bind_coll(pybind11::module_& m);

} // namespace cclx_ops
