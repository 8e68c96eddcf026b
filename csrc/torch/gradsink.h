// Gradients that go straight into a parameter's .grad.
//
// A data-parallel wrapper keeps .grad of every parameter as a view of a flat bucket.  Handing autograd a fresh gradient per
// parameter then costs an allocation, a launch and a pass over memory per parameter to add it to the bucket; the nodes of
// this binding add there themselves (a matrix product with beta = 1, or a kernel that accumulates).  They do so only when the
// wrapper asked for it (`grad_sink` of the module), in a plain backward() call (not autograd.grad or backward(inputs=...),
// whose callers want the gradients returned, nor with create_graph), for parameters without hooks of any kind (with several
// ranks the wrapper has hooks on all of them, and autograd delivers), and on the stream autograd would have used and made
// the caller wait for.
#pragma once

#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/variable.h>

#include "common.h"

namespace mccl_torch {

class GradSink {
 public:
  explicit GradSink(bool on) {
    if (!on || at::GradMode::is_enabled()) return;
    const auto* info = torch::autograd::get_current_graph_task_exec_info();
    direct_ = info == nullptr || info->empty();
  }
  // The buffer to add p's gradient to; undefined where it has to be returned instead.
  Tensor buffer(const Tensor& p) const {
    namespace impl = torch::autograd::impl;
    if (!direct_ || !p.requires_grad() || !p.is_leaf() || !impl::hooks(p).empty() || impl::post_acc_grad_hooks(p) != nullptr) return Tensor();
    const Tensor& g = p.grad();
    if (!g.defined() || g.requires_grad() || g.scalar_type() != p.scalar_type() || g.sizes() != p.sizes() || !g.is_contiguous() || !aligned16(g))
      return Tensor();
    const auto acc = impl::grad_accumulator(p);
    if (!acc->post_hooks().empty() || !acc->pre_hooks().empty()) return Tensor();
    const auto stream = acc->stream();
    if (stream && *stream != c10::cuda::getCurrentCUDAStream(p.device().index()).unwrap()) return Tensor();
    return g;
  }

 private:
  bool direct_ = false;
};

// d p += dy^T x, into the buffer or into *ret; nothing for a frozen weight.
inline void weightGrad(GradSink& sink, const Tensor& p, const Tensor& dy, const Tensor& x, Tensor* ret) {
  if (!p.requires_grad()) return;
  Tensor g = sink.buffer(p);
  if (g.defined()) at::addmm_out(g, g, dy.t(), x); else *ret = at::mm(dy.t(), x);
}

// Where kernels put the gradients of several vectors at once: all of them into their buffers, or all into new tensors.
struct VectorGrads {
  Tensor t[3];
  bool direct = true;
  VectorGrads(GradSink& sink, std::initializer_list<const Tensor*> params) {
    int n = 0;
    for (const Tensor* p : params) { t[n] = sink.buffer(*p); direct = direct && t[n].defined(); ++n; }
    n = 0;
    for (const Tensor* p : params) { if (!direct) t[n] = at::empty(p->sizes(), p->options()); ++n; }
  }
  Tensor ret(int i) const { return direct ? Tensor() : t[i]; }
};

}  // namespace mccl_torch
