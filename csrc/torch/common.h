// Shared by the torch binding's translation units: tensor to pointer, stream and status helpers.
//
// The binding exists for the host side of the small calls: an entry point that checks its arguments, allocates its outputs,
// launches and records its autograd node in C++ costs a few microseconds where the same steps through ctypes and a Python
// autograd.Function cost tens.  It holds no kernels of its own: everything it launches is libmccl's C API or an ATen
// operator.
#pragma once

#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <ATen/cuda/CUDAContextLight.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>

#include "mccl.h"
#include "mccl_ops.h"

namespace mccl_torch {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// Kernels of this library launched through the binding, by the module that reports them.
struct Counters { std::atomic<int64_t> norm{0}, loss{0}, optim{0}, gemm{0}, moe{0}; };
inline Counters& counters() { static Counters c; return c; }

inline mcclStream_t streamOf(const Tensor& t) {
  return reinterpret_cast<mcclStream_t>(c10::cuda::getCurrentCUDAStream(t.device().index()).stream());
}
inline void check(mcclResult_t rc, const char* what) {
  TORCH_CHECK(rc == mcclSuccess || rc == mcclInProgress, "mccl: ", mcclResultStr(rc), " (code ", (int)rc, "): ", what);
}
inline bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }
// Widths at which LayerNorm runs in the library's kernels (FusedLayerNorm and the decoder's nodes alike).  The kernels take
// others too, in another order of their sums than the tensor library's: a model's results would depend on it.
inline bool layerNormWidth(int64_t d) { return d == 256 || d == 512 || d == 1024; }
inline bool bf16Cuda(const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kBFloat16; }

// Whether a kernel may be launched on t's memory in place of tensor operations: not for the wrappers of torch.func, of tensor
// subclasses and of tracing, nor for a tensor with a forward-mode tangent; what sees them has to see operators.
inline bool ordinary(const Tensor& t) {
  constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                         c10::DispatchKey::Functionalize});
  return t.defined() && t.has_storage() && !t.key_set().has_any(wrapped) && !t._fw_grad(0).defined();
}
// A trace or a dispatch mode records operators: the nodes stand aside for it.
inline bool recorded() { return torch::jit::tracer::isTracing() || c10::impl::TorchDispatchModeTLS::any_modes_set(); }

// For the inside of a node: operators record no gradient and keep the types they are given, whatever autocast says.
struct Below {
  at::AutoDispatchBelowADInplaceOrView noGrad;
  c10::impl::ExcludeDispatchKeyGuard noCast{c10::autocast_dispatch_keyset};
};

// Gradients that have no graph of their own: differentiating them (backward(create_graph=True)) raises instead of counting
// them as constants.
inline variable_list once(variable_list&& grads) {
  if (!at::GradMode::is_enabled()) return std::move(grads);
  auto raise = std::make_shared<torch::autograd::DelayedError>("mccl: the gradient of a fused node cannot be differentiated again", (int64_t)grads.size());
  for (Tensor& g : grads) if (g.defined()) g = g.detach().requires_grad_(true);
  return raise->apply(std::move(grads));
}

// One module's functions each, defined in the files of the same names.
void bindOps(pybind11::module_& m);
void bindComm(pybind11::module_& m);
void bindMoe(pybind11::module_& m);
void bindGpt2(pybind11::module_& m);
void bindLlama(pybind11::module_& m);

}  // namespace mccl_torch
