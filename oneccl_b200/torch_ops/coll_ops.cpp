// Host side of the small calls on a device group and of the expert-parallel steps: tensors to pointer tables without a
// Python loop over them (kernels: csrc/gpu/launch_allreduce.cu, moe_kernels.cu).  A launch into a full queue waits for the GPU:
// other Python threads run meanwhile.
#include "torch_ops.hpp"

namespace cclx_ops {
namespace {

typedef std::vector<Tensor> tensors;

int ccl_dtype(at::ScalarType t) {
    switch (t) {
        case at::kChar: return 0;
        case at::kByte:
        case at::kBool: return 1;
        case at::kShort: return 2;
        case at::kUInt16: return 3;
        case at::kInt: return 4;
        case at::kUInt32: return 5;
        case at::kLong: return 6;
        case at::kUInt64: return 7;
        case at::kHalf: return 8;
        case at::kFloat: return 9;
        case at::kDouble: return 10;
        case at::kBFloat16: return 11;
        default: throw pybind11::type_error(std::string(c10::toString(t)) + " has no ccl datatype");
    }
}

template <class T>
std::vector<T*> pointers(const tensors& ts) {
    std::vector<T*> p;
    p.reserve(ts.size());
    for (const auto& t : ts)
        p.push_back(reinterpret_cast<T*>(t.data_ptr()));
    return p;
}

// one tensor per entry: this rank's, or one per emulated rank
void allreduce(uintptr_t group, const tensors& send, const tensors& recv, int op, int algo, int blocks, std::optional<double> scale,
               std::optional<uintptr_t> stream) {
    for (size_t i = 0; i < send.size(); i++)
        if (!send[i].is_contiguous() || !recv[i].is_contiguous() || send[i].numel() != recv[i].numel()) {
            PyErr_SetString(PyExc_AssertionError, "allreduce takes contiguous tensors of one size");
            throw pybind11::error_already_set();
        }
    void* st = stream ? reinterpret_cast<void*>(*stream) : stream_of(send[0]);
    const auto s = pointers<const void>(send);
    const auto r = pointers<void>(recv);
    const int dt_in = ccl_dtype(send[0].scalar_type()), dt_out = ccl_dtype(recv[0].scalar_type());
    pybind11::gil_scoped_release nogil;
    check(cclx_dc_allreduce(reinterpret_cast<void*>(group), s.data(), r.data(), send[0].numel(), dt_in, dt_out, op, algo, blocks,
                            scale ? (float)*scale : 1.0f, scale ? 1 : 0, st));
}

// expert ids [T, k], weights [T, k], items per expert [E], grouping permutation and its inverse [T * k]
pybind11::tuple route(const Tensor& logits_, int64_t topk) {
    const Tensor logits = logits_.scalar_type() == at::kFloat && logits_.is_contiguous() ? logits_ : logits_.to(at::kFloat).contiguous();
    const int64_t T = logits.size(0), E = logits.size(1);
    // 16-byte aligned parts: ids, order, places, weights, counts; the cursors lie right behind the counts
    const int64_t n = T * topk;
    const size_t items = ((size_t)n * 8 + 15) / 16 * 16, w_at = 3 * items, c_at = w_at + ((size_t)n * 4 + 15) / 16 * 16;
    const Tensor all = empty_on(logits, { (int64_t)c_at + 12 * E }, at::kByte);
    char* base = static_cast<char*>(all.data_ptr());
    auto longs = [&](size_t at) { return reinterpret_cast<long long*>(base + at); };
    {
        pybind11::gil_scoped_release nogil;
        check(cclx_moe_route(logits.data_ptr<float>(), (int)T, (int)E, (int)topk, longs(0), reinterpret_cast<float*>(base + w_at),
                             longs(c_at), longs(items), longs(2 * items), longs(c_at) + E, stream_of(logits)));
    }
    return pybind11::make_tuple(part_of(all, 0, { T, topk }, at::kLong), part_of(all, w_at, { T, topk }, at::kFloat),
                                part_of(all, c_at, { E }, at::kLong), part_of(all, items, { n }, at::kLong),
                                part_of(all, 2 * items, { n }, at::kLong));
}

void dispatch(uintptr_t group, const tensors& x, const tensors& order, const tensors& counts, const tensors& meta, const Tensor& recv,
              const Tensor& table, int topk, int blocks) {
    const auto px = pointers<const void>(x);
    const auto po = pointers<const long long>(order), pc = pointers<const long long>(counts);
    const auto pm = pointers<int>(meta);
    pybind11::gil_scoped_release nogil;
    check(cclx_moe_dispatch(reinterpret_cast<void*>(group), px.data(), po.data(), pc.data(), pm.data(), order[0].numel(), topk,
                            (int)x[0].size(1), recv.data_ptr(), recv.size(0), table.data_ptr(), blocks, stream_of(recv)));
}

void combine(uintptr_t group, const tensors& expert, const tensors& pos, const tensors& weight, const tensors& out, const tensors& meta,
             const Tensor& expert_out, int topk, int blocks) {
    const auto pe = pointers<const long long>(expert), pp = pointers<const long long>(pos);
    const auto pw = pointers<const float>(weight);
    const auto po = pointers<void>(out);
    const auto pm = pointers<int>(meta);
    pybind11::gil_scoped_release nogil;
    check(cclx_moe_combine_peer(reinterpret_cast<void*>(group), pe.data(), pp.data(), pw.data(), po.data(), pm.data(),
                                expert[0].numel(), topk, (int)out[0].size(1), expert_out.data_ptr(), blocks,
                                stream_of(expert_out)));
}

} // namespace

void bind_coll(pybind11::module_& m) {
    m.def("dc_allreduce", &allreduce);
    m.def("moe_route", &route);
    m.attr("route_one_block") = cclx_moe_route_one_block();
    m.def("moe_dispatch", &dispatch);
    m.def("moe_combine", &combine);
}

} // namespace cclx_ops
