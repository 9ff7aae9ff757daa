// Host runtime of the package: the per-call work around the C ABI (argument checks, allocation, autograd bookkeeping,
// launch order) as native code.  A small scan is five kernels of 2..10 us; driven from Python its call took 170 us, of
// which the interpreter, ctypes and the hand-over of the GIL to autograd's worker thread were about 110.
#pragma once
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>

#include "qllm2_pam.h"

namespace qhost {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// qllm2_b200._lib.QPamError in Python: by the module's exception translator in a call, by torch's from a backward pass.
struct Error : torch::PyTorchError {
  using PyTorchError::PyTorchError;
  PyObject* python_type() override;
};

template <typename... Args>
[[noreturn]] inline void fail(const Args&... args) {
  throw Error(c10::str(args...));
}
#define QH_REQUIRE(cond, ...)                  \
  do {                                         \
    if (!(cond)) ::qhost::fail(__VA_ARGS__);   \
  } while (0)

inline void check(int rc, const char* what) {
  if (rc != 0) fail(what, " failed with code ", rc, ": ", qpam_last_error());
}

inline void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
inline Tensor value(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

inline int dtype_code(at::ScalarType t) {
  if (t == at::kFloat) return QPAM_F32;
  if (t == at::kBFloat16) return QPAM_BF16;
  fail("unsupported dtype ", t, ": the PAM kernels take float32 or bfloat16");
}
inline Tensor workspace(size_t bytes, const Tensor& like) {
  return at::empty({(int64_t)std::max<size_t>(bytes, 256)}, like.options().dtype(at::kByte));
}
// Contiguous and starting on a boundary of `align` bytes, as the kernels' vector accesses need it (a view into a flat buffer may
// start anywhere).  Differentiable like the copies it is made of.
inline Tensor dense(const Tensor& t, size_t align = 16) {
  const Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % align ? c.clone() : c;
}
// Token tensors: whole complex numbers at least.  (Off a 16-byte boundary the scan takes them through its scalar kernels.)
inline Tensor dense_tokens(const Tensor& t) { return dense(t, 2 * t.element_size()); }
inline bool needs_grad(const Tensor& t) { return t.defined() && t.requires_grad(); }
inline std::string shape(const Tensor& t) { return c10::str(t.sizes()); }

inline bool autocast_bf16() {
  return at::autocast::is_autocast_enabled(at::kCUDA) && at::autocast::get_autocast_dtype(at::kCUDA) == at::kBFloat16;
}

// Descriptor of a packed batch (int32 [S+1]) on the tokens' device; a host descriptor is checked here (the kernels check a
// device descriptor themselves and report through the status word).
Tensor descriptor(const Tensor& cu, int64_t T, at::Device device);

// Forward scan with token-major output [B,T,H*d,2] and the final states [K,S,H,d,d,2]; inputs contiguous, of the scan's dtypes.
std::tuple<Tensor, Tensor> scan_tokens(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const Tensor& coef, const Tensor& s0,
                                       const Tensor& cu, double q_scale);

// The same with the final states going straight to the slots of a state pool; false where the kernels do not offer it.
bool scan_prefill(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const Tensor& coef, const Tensor& s0, const Tensor& cu, double q_scale,
                  const Tensor& pool, const Tensor& slots, int64_t layer, Tensor& y);

void bind_scan(pybind11::module_& m);
void bind_loss(pybind11::module_& m);
void bind_forward(pybind11::module_& m);
void bind_block(pybind11::module_& m);

}  // namespace qhost
