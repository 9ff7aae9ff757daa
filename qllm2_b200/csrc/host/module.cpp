#include "common.h"

namespace py = pybind11;

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const qhost::Error& e) {
      py::object cls = py::module_::import("qllm2_b200._lib").attr("QPamError");
      PyErr_SetString(cls.ptr(), e.what());
    }
  });
  qhost::bind_scan(m);
  qhost::bind_loss(m);
  qhost::bind_forward(m);
  qhost::bind_block(m);
}
