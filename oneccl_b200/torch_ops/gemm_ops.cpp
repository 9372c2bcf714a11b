// Host side of the plain bf16 product (kernels: csrc/gpu/gemm_small.cu, gemm_2sm.cu, fused_gemm.cuh).
#include "torch_ops.hpp"

namespace cclx_ops {
namespace {

// kernel: 0 = the library decides, 1 = one CTA per tile, 2 = CTA pairs
Tensor gemm_bf16(const Tensor& a_, const Tensor& w_, const std::optional<Tensor>& out_, int64_t epilogue, int64_t ctas, int64_t kernel,
                 const std::optional<Tensor>& rows, const Tensor& err) {
    pybind11::gil_scoped_release nogil;
    const Tensor a = a_.is_contiguous() ? a_ : a_.contiguous(), w = w_.is_contiguous() ? w_ : w_.contiguous();
    const int M = (int)a.size(0), K = (int)a.size(1), N = (int)w.size(0);
    const Tensor out = out_ ? *out_ : empty_on(a, { M, N }, at::kBFloat16);
    void* st = stream_of(a);
    if (rows)
        check(cclx_gemm_bf16_rows(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, (int)epilogue, rows->data_ptr(),
                                  err.data_ptr(), st));
    else if (kernel == 2)
        check(cclx_gemm_bf16_2sm(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, (int)epilogue, (int)ctas / 2,
                                 err.data_ptr(), st));
    else
        check(cclx_gemm_bf16(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, (int)epilogue,
                             kernel == 1 ? -((int)ctas + 1) : (int)ctas, err.data_ptr(), st));
    return out;
}

} // namespace

void bind_gemm(pybind11::module_& m) {
    m.def("gemm_bf16", &gemm_bf16);
}

} // namespace cclx_ops
