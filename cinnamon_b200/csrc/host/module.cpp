// Python module of the native host path: function pointers in, differentiable calls out.
#include "host.h"

namespace cinnhost {
Api api;
PyObject* library_error = PyExc_RuntimeError;
void bind_linear(pybind11::module_& m);
void bind_attention(pybind11::module_& m);
void bind_moe(pybind11::module_& m);
void bind_moe_train(pybind11::module_& m);
}  // namespace cinnhost

PYBIND11_MODULE(_host, m) {
    using namespace cinnhost;
    m.def("bind", [](const std::unordered_map<std::string, uintptr_t>& addr, pybind11::object error_type) {
        library_error = error_type.release().ptr();        // (bound once, kept for the life of the process)
#define CINN_BIND(name) api.name = reinterpret_cast<decltype(api.name)>(addr.at(#name));
        CINN_HOST_API(CINN_BIND)
#undef CINN_BIND
    });
    m.def("symbols", [] {
        std::vector<std::string> names;
#define CINN_NAME(name) names.push_back(#name);
        CINN_HOST_API(CINN_NAME)
#undef CINN_NAME
        return names;
    });
    pybind11::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const CinnError& e) {
            PyErr_SetString(e.invalid ? PyExc_AssertionError : library_error, e.what());
        }
    });
    bind_linear(m);
    bind_attention(m);
    bind_moe(m);
    bind_moe_train(m);
}
