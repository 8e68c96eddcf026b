// Gradients that go straight into a parameter's .grad.
//
// A data-parallel wrapper keeps .grad of every parameter as a view of a flat bucket.  Handing autograd a fresh gradient per
// parameter then costs an allocation, a launch and a pass over memory per parameter to add it to the bucket; the nodes of
// this binding add there themselves (a matrix product with beta = 1, or a kernel that accumulates).  They do so only when the
// wrapper asked for it (a sink number on the module), in a plain backward() call (not autograd.grad or backward(inputs=...),
// whose callers want the gradients returned), and for parameters without hooks of the user's.
#pragma once

#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/variable.h>

#include "common.h"

namespace mccl_torch {

// Sink numbers: 0 none, -1 accumulate, > 0 accumulate and call the registered Python function with the parameter.
class GradSink {
 public:
  GradSink(int64_t id) : id_(id) {
    if (id == 0) return;
    const auto* info = torch::autograd::get_current_graph_task_exec_info();
    direct_ = info == nullptr || info->empty();
  }
  // The buffer to add p's gradient to; undefined where it has to be returned instead.
  Tensor buffer(const Tensor& p) const {
    if (!direct_ || !p.requires_grad() || !p.is_leaf() || !torch::autograd::impl::hooks(p).empty()) return Tensor();
    const Tensor& g = p.grad();
    if (!g.defined() || g.requires_grad() || g.scalar_type() != p.scalar_type() || g.sizes() != p.sizes() || !g.is_contiguous() || !aligned16(g))
      return Tensor();
    return g;
  }
  // `p` has received all of its gradient.
  void done(const Tensor& p) { if (id_ > 0) done_.push_back(p); }
  // Tells the wrapper; once, after the node's launches.
  void flush();

 private:
  int64_t id_;
  bool direct_ = false;
  std::vector<Tensor> done_;
};

// d p += dy^T x, into the buffer or into *ret.
inline void weightGrad(GradSink& sink, const Tensor& p, const Tensor& dy, const Tensor& x, Tensor* ret, bool last = true) {
  Tensor g = sink.buffer(p);
  if (!g.defined()) { *ret = at::mm(dy.t(), x); return; }
  at::addmm_out(g, g, dy.t(), x);
  if (last) sink.done(p);
}

// Where kernels put the gradients of several vectors at once: all of them into their buffers, or all into new tensors.
struct VectorGrads {
  Tensor t[3];
  bool direct = true;
  VectorGrads(GradSink& sink, std::initializer_list<const Tensor*> params) {
    int n = 0;
    for (const Tensor* p : params) { t[n] = sink.buffer(*p); direct = direct && t[n].defined(); ++n; }
    n = 0;
    for (const Tensor* p : params) { if (direct) sink.done(*p); else t[n] = at::empty(p->sizes(), p->options()); ++n; }
  }
  Tensor ret(int i) const { return direct ? Tensor() : t[i]; }
};

}  // namespace mccl_torch
