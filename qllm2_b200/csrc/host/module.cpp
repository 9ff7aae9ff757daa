#include "common.h"

namespace py = pybind11;

PyObject* qhost::Error::python_type() { return py::module_::import("qllm2_b200._lib").attr("QPamError").ptr(); }   // (the module keeps it)

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (qhost::Error& e) {
      PyErr_SetString(e.python_type(), e.what());
    }
  });
  qhost::bind_scan(m);
  qhost::bind_loss(m);
  qhost::bind_forward(m);
  qhost::bind_block(m);
}
