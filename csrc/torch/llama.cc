// Nodes of the Llama style decoder on a communicator of one rank: the two halves of a block around attention and the final
// norm.  As in gpt2.cc the residual add belongs to the norm behind it.  RMSNorm, rotation and SwiGLU ran as fp32 tensor
// operations before (about 190 launches forward and backward per block, most of them over fp32 copies of the activations).
#include "nodes.h"

namespace mccl_torch {
namespace {

Tensor rmsStats(const Tensor& x, int64_t rows) { return at::empty({rows}, x.options().dtype(at::kFloat)); }

// sum = x + pending (pending may be null: sum = x), h = RMSNorm(sum) * w.
void addRms(const Tensor& x, const Tensor* pending, const Tensor& w, double eps, Tensor* sum, Tensor* h, Tensor* rstd) {
  const int64_t T = x.size(0), d = x.size(1);
  *rstd = rmsStats(x, T);
  *h = at::empty({T, d}, x.options());
  *sum = pending ? at::empty({T, d}, x.options()) : at::alias(x);
  check(mcclRmsNormForward(x.data_ptr(), pending ? pending->data_ptr() : nullptr, w.data_ptr(), pending ? sum->data_ptr() : nullptr, h->data_ptr(),
                           rstd->data_ptr<float>(), T, (int)d, (float)eps, streamOf(x)), "mcclRmsNormForward");
  counters().norm++;
}

// Gradient of the sum from those of h (up to three parts, added up on the way where there is a residual stream) and, where
// defined, of the residual stream.
Tensor addRmsBackward(const Tensor& sum, std::initializer_list<Tensor> parts, const Tensor& dres, const Tensor& w, const Tensor& rstd, GradSink& sink, Tensor* dw) {
  const int64_t T = sum.size(0), d = sum.size(1);
  Tensor dx = at::empty({T, d}, sum.options());
  Tensor partial = at::empty({(int64_t)mcclLayerNormPartials(T) * d}, rstd.options());
  Tensor res = dres.defined() ? rows2d(dres, T, d) : Tensor();
  const void* dh[3] = {};
  int n = 0;
  for (const Tensor& p : parts) dh[n++] = p.data_ptr();
  VectorGrads g(sink, {&w});
  check(mcclRmsNormBackward(sum.data_ptr(), dh[0], dh[1], dh[2], res.defined() ? res.data_ptr() : nullptr, w.data_ptr(), rstd.data_ptr<float>(),
                            dx.data_ptr(), g.t[0].data_ptr(), g.direct, partial.data_ptr<float>(), T, (int)d, streamOf(sum)), "mcclRmsNormBackward");
  counters().norm += 2;
  *dw = g.ret(0);
  return dx;
}

// The gradients of q and k turned back, as [T, d]; any strides with adjacent elements of a head.
void unrotate(const Tensor& dq, const Tensor& dk, int64_t T, int64_t d, double theta, Tensor* oq, Tensor* ok) {
  auto fits = [](const Tensor& t) { return t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 && aligned16(t); };
  Tensor q = fits(dq) ? dq : dq.contiguous(), k = fits(dk) ? dk : dk.contiguous();
  *oq = at::empty({T, d}, q.options());
  *ok = at::empty({T, d}, q.options());
  const int b = (int)q.size(0), h = (int)q.size(1), s = (int)q.size(2), hd = (int)q.size(3);
  if (q.strides() == k.strides()) {
    check(mcclRope(q.data_ptr(), k.data_ptr(), oq->data_ptr(), ok->data_ptr(), b, s, h, hd, q.stride(0), q.stride(2), q.stride(1), (float)theta, 1,
                   streamOf(q)), "mcclRope");
    return;
  }
  check(mcclRope(q.data_ptr(), nullptr, oq->data_ptr(), nullptr, b, s, h, hd, q.stride(0), q.stride(2), q.stride(1), (float)theta, 1, streamOf(q)), "mcclRope");
  check(mcclRope(k.data_ptr(), nullptr, ok->data_ptr(), nullptr, b, s, h, hd, k.stride(0), k.stride(2), k.stride(1), (float)theta, 1, streamOf(k)), "mcclRope");
}

struct LlamaInFn : torch::autograd::Function<LlamaInFn> {
  // Outputs: residual [T, d], q and k (rotated) and v as [b, h, s, hd].
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& pending, const Tensor& nw, const Tensor& wq, const Tensor& wk,
                               const Tensor& wv, int64_t b, int64_t s, int64_t heads, double theta, double eps, bool sink) {
    Below below;
    const int64_t T = x.size(0), d = x.size(1), hd = d / heads;
    Tensor sum, h, rstd;
    addRms(x, pending ? &*pending : nullptr, nw, eps, &sum, &h, &rstd);
    Tensor q = at::linear(h, wq), k = at::linear(h, wk), v = at::linear(h, wv);
    check(mcclRope(q.data_ptr(), k.data_ptr(), q.data_ptr(), k.data_ptr(), (int)b, (int)s, (int)heads, (int)hd, s * d, d, hd, (float)theta, 0,
                   streamOf(x)), "mcclRope");
    auto split = [&](const Tensor& t) { return t.as_strided({b, heads, s, hd}, {s * d, hd, d, 1}); };
    ctx->save_for_backward({pending ? sum : x, h, rstd, nw, wq, wk, wv});      // the input itself: a change in place is noticed
    ctx->saved_data["sink"] = sink;
    ctx->saved_data["theta"] = theta;
    ctx->saved_data["pending"] = pending.has_value();
    return {sum, split(q), split(k), split(v)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &sum = saved[0], &h = saved[1], &rstd = saved[2], &nw = saved[3], &wq = saved[4], &wk = saved[5], &wv = saved[6];
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = h.size(0), d = h.size(1);
    variable_list ret(12);
    Tensor dq, dk, dv = fromHeads(g[3], T, d);
    unrotate(g[1], g[2], T, d, ctx->saved_data["theta"].toDouble(), &dq, &dk);
    Tensor dhv = at::mm(dv, wv), dhk = at::mm(dk, wk), dhq = at::mm(dq, wq);
    weightGrad(sink, wv, dv, h, &ret[5]);
    weightGrad(sink, wk, dk, h, &ret[4]);
    weightGrad(sink, wq, dq, h, &ret[3]);
    Tensor dx = addRmsBackward(sum, {dhv, dhk, dhq}, g[0], nw, rstd, sink, &ret[2]);
    ret[0] = dx;
    if (ctx->saved_data["pending"].toBool()) ret[1] = dx;
    return once(std::move(ret));
  }
};

struct LlamaOutFn : torch::autograd::Function<LlamaOutFn> {
  // Outputs: residual after attention, MLP output, both [T, d].
  static variable_list forward(AutogradContext* ctx, const Tensor& a, const Tensor& res, const Tensor& wo, const Tensor& nw, const Tensor& wg,
                               const Tensor& wu, const Tensor& wd, double eps, bool sink) {
    Below below;
    const int64_t T = res.size(0), d = res.size(1);
    Tensor a2 = fromHeads(a, T, d), p = at::linear(a2, wo), x1, h, rstd;
    addRms(res, &p, nw, eps, &x1, &h, &rstd);
    Tensor gate = at::linear(h, wg), up = at::linear(h, wu), act = at::empty(gate.sizes(), gate.options());
    check(mcclSwigluForward(gate.data_ptr(), up.data_ptr(), act.data_ptr(), act.numel(), streamOf(act)), "mcclSwigluForward");
    Tensor y = at::linear(act, wd);
    ctx->save_for_backward({a2, x1, h, rstd, gate, up, wo, nw, wg, wu, wd});
    ctx->saved_data["sink"] = sink;
    ctx->saved_data["b"] = a.size(0);
    ctx->saved_data["h"] = a.size(1);
    return {x1, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &a2 = saved[0], &x1 = saved[1], &h = saved[2], &rstd = saved[3], &gate = saved[4], &up = saved[5], &wo = saved[6], &nw = saved[7],
                 &wg = saved[8], &wu = saved[9], &wd = saved[10];
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = h.size(0), d = h.size(1), b = ctx->saved_data["b"].toInt(), heads = ctx->saved_data["h"].toInt();
    variable_list ret(9);
    Tensor dy = rows2d(g[1], T, d);
    Tensor dact = at::mm(dy, wd);
    // The product is worked out again from gate and up: the pass reads both anyway, and it need not be kept.
    Tensor act = at::empty(gate.sizes(), gate.options()), dgate = at::empty(gate.sizes(), gate.options());
    Tensor dup = dact;
    check(mcclSwigluBackward(gate.data_ptr(), up.data_ptr(), dact.data_ptr(), act.data_ptr(), dgate.data_ptr(), dup.data_ptr(), act.numel(),
                             streamOf(act)), "mcclSwigluBackward");
    weightGrad(sink, wd, dy, act, &ret[6]);
    Tensor dhu = at::mm(dup, wu), dhg = at::mm(dgate, wg);
    weightGrad(sink, wg, dgate, h, &ret[4]);
    weightGrad(sink, wu, dup, h, &ret[5]);
    Tensor dx = addRmsBackward(x1, {dhu, dhg}, g[0], nw, rstd, sink, &ret[3]);
    Tensor da = at::mm(dx, wo);
    weightGrad(sink, wo, dx, a2, &ret[2]);
    ret[0] = da.view({b, T / b, heads, d / heads}).transpose(1, 2);
    ret[1] = dx;
    return once(std::move(ret));
  }
};

struct FinalRmsFn : torch::autograd::Function<FinalRmsFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& pending, const Tensor& w, double eps, bool sink) {
    Below below;
    Tensor sum, h, rstd;
    addRms(x, &pending, w, eps, &sum, &h, &rstd);
    ctx->save_for_backward({sum, rstd, w});
    ctx->saved_data["sink"] = sink;
    return h;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    Below below;
    c10::cuda::CUDAGuard guard(saved[0].device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    variable_list ret(5);
    Tensor dx = addRmsBackward(saved[0], {rows2d(g[0], saved[0].size(0), saved[0].size(1))}, Tensor(), saved[2], saved[1], sink, &ret[2]);
    ret[0] = dx;
    ret[1] = dx;
    return once(std::move(ret));
  }
};

// One block on x + pending (both [T, d]; pending may be missing).  p: norm1, q, k, v, o, norm2, gate, up, down.  Returns two
// tensors whose sum is the block's output, or None where the kernels do not cover the case.
py::object block(const Tensor& x, const OptTensor& pending, const std::vector<Tensor>& p, int64_t b, int64_t s, int64_t heads, double theta,
                 double eps, bool sink) {
  if (p.size() != 9 || x.dim() != 2 || !usable(x, p) || !attentionOnce()) return py::none();
  const int64_t d = x.size(1), f = p[6].size(0);
  if (heads <= 0 || d % heads || (d / heads) % 16 || x.size(0) != b * s) return py::none();
  if (pending && (!plainBf16(*pending, x) || !shaped(*pending, x.sizes()))) return py::none();
  if (!shaped(p[0], {d}) || !shaped(p[5], {d}) || !shaped(p[6], {f, d}) || !shaped(p[7], {f, d}) || !shaped(p[8], {d, f})) return py::none();
  for (int i = 1; i < 5; ++i) if (!shaped(p[i], {d, d})) return py::none();
  c10::cuda::CUDAGuard guard(x.device());
  variable_list in = LlamaInFn::apply(x, pending, p[0], p[1], p[2], p[3], b, s, heads, theta, eps, sink);
  Tensor a = at::scaled_dot_product_attention(in[1], in[2], in[3], {}, 0.0, true);
  variable_list out = LlamaOutFn::apply(a, in[0], p[4], p[5], p[6], p[7], p[8], eps, sink);
  return py::make_tuple(out[0], out[1]);
}

py::object finalRms(const Tensor& x, const Tensor& pending, const Tensor& w, double eps, bool sink) {
  if (!usable(x, {pending, w}) || x.dim() != 2 || !shaped(pending, x.sizes()) || !shaped(w, {x.size(1)})) return py::none();
  c10::cuda::CUDAGuard guard(x.device());
  return py::cast(FinalRmsFn::apply(x, pending, w, eps, sink));
}

}  // namespace

void bindLlama(py::module_& m) {
  m.def("llama_block", &block);
  m.def("llama_final_norm", &finalRms);
}

}  // namespace mccl_torch
