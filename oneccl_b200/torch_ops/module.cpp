#include "torch_ops.hpp"

namespace cclx_ops {
std::atomic<long long> launches{ 0 };
std::atomic<int> GradSink::live{ 0 };

SinkRef sink_of(const pybind11::object& param) {
    if (GradSink::live.load(std::memory_order_relaxed) == 0 || param.is_none())
        return nullptr;
    static PyObject* name = PyUnicode_InternFromString("_grad_sink");
    PyObject* s = PyObject_GetAttr(param.ptr(), name);
    if (!s) {
        PyErr_Clear();
        return nullptr;
    }
    return pybind11::reinterpret_steal<pybind11::object>(s).cast<SinkRef>();
}
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    using namespace cclx_ops;
    namespace py = pybind11;
    // released by the interpreter's end: the translator below may run as long as the interpreter does
    static PyObject* error_type = py::object(py::module_::import("oneccl_b200._lib").attr("CclError")).release().ptr();
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p)
                std::rethrow_exception(p);
        }
        catch (const ccl_error& e) {
            PyErr_SetString(error_type, e.what());
        }
    });
    m.def("launch_count", [] { return launches.load(); });
    m.def("stream_ptr", [] {
        const auto s = at::cuda::getCurrentCUDAStream();
        set_device(s.device_index());
        return reinterpret_cast<uintptr_t>(s.stream());
    }, "handle of the current stream; the library's runtime follows its device");
    m.def("set_device", [](int dev) { set_device(dev); });
    py::class_<GradStream, GradStreamRef>(m, "GradStream")
        .def(py::init<int>())
        .def("join", [](GradStream& g, uintptr_t stream, int dev) {
            g.join(at::cuda::getStreamFromExternal(reinterpret_cast<cudaStream_t>(stream), (c10::DeviceIndex)dev));
        })
        .def("finish", &GradStream::finish)
        .def_property_readonly("handle", &GradStream::handle);
    py::class_<GradSink, SinkRef>(m, "GradSink")
        .def(py::init<Tensor, py::object>())
        .def_readonly("grad", &GradSink::grad)
        .def_readwrite("fresh", &GradSink::fresh)
        .def("begin_step", [](GradSink& s, const GradStreamRef& beside) {
            s.fresh = true;
            s.on_side = false;
            s.beside = beside;
        })
        // whether the parameter received a gradient since begin_step
        .def("end_step", [](GradSink& s) {
            const bool got = !s.fresh;
            s.fresh = s.on_side = false;
            s.beside = nullptr;
            return got;
        })
        // gradients that autograd accumulates itself are added in place: give them a clean buffer first
        .def("clear_before_accumulation",
             [](const SinkRef& s, const Tensor& param) {
                 std::weak_ptr<GradSink> w = s;
                 return param.register_hook([w](const Tensor& g) {
                     if (const SinkRef s = w.lock(); s && g.defined() && !s->add())
                         s->grad.zero_();
                 });
             })
        .def("remove_hook", [](const SinkRef&, const Tensor& param, unsigned h) { param.remove_hook(h); });
    bind_nn(m);
    bind_train(m);
    bind_gemm(m);
    bind_coll(m);
}
