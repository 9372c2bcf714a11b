#include "torch_ops.hpp"

namespace cclx_ops {
std::atomic<long long> launches{ 0 };
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
    bind_nn(m);
    bind_train(m);
    bind_gemm(m);
}
