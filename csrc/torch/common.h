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
inline bool bf16Cuda(const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kBFloat16; }

// One module's functions each, defined in the files of the same names.
void bindOps(pybind11::module_& m);
void bindComm(pybind11::module_& m);
void bindMoe(pybind11::module_& m);
void bindGpt2(pybind11::module_& m);
void bindLlama(pybind11::module_& m);

}  // namespace mccl_torch
