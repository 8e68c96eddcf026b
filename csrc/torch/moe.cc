// Mixture-of-experts layer of the torch binding: the routing as an autograd node, and the whole layer as one node when every
// expert lives on this GPU.
#include "common.h"

namespace mccl_torch {
namespace {

struct Routed { Tensor gate, lse, flat, inverse, kept; };

Routed route(const Tensor& logits, int64_t capacity, bool slots) {
  const int64_t T = logits.size(0), E = logits.size(1);
  Routed r;
  auto f32 = logits.options().dtype(at::kFloat), i32 = logits.options().dtype(at::kInt);
  Tensor stats = at::empty({2, T}, f32);
  r.gate = stats.select(0, 0);
  r.lse = stats.select(0, 1);
  const int64_t scratch = mcclMoeRouteScratch((int)T, (int)E);
  Tensor ints = at::empty({T + (slots ? E * capacity + E : 0) + scratch}, i32);
  r.flat = ints.narrow(0, 0, T);
  if (slots) {
    r.inverse = ints.narrow(0, T, E * capacity);
    r.kept = ints.narrow(0, T + E * capacity, E);
  }
  int32_t* base = ints.data_ptr<int32_t>();
  check(mcclMoeRoute(logits.data_ptr(), (int)T, (int)E, (int)capacity, r.gate.data_ptr<float>(), r.lse.data_ptr<float>(), base,
                     slots ? base + T : nullptr, slots ? base + T + E * capacity : nullptr, base + ints.numel() - scratch, streamOf(logits)),
        "mcclMoeRoute");
  counters().moe += 2;
  return r;
}

struct RouteFn : torch::autograd::Function<RouteFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& logits, int64_t capacity) {
    c10::cuda::CUDAGuard guard(logits.device());
    Tensor l = logits.contiguous();
    Routed r = route(l, capacity, false);
    ctx->save_for_backward({l, r.lse, r.flat});
    ctx->saved_data["capacity"] = capacity;
    ctx->mark_non_differentiable({r.flat});
    return {r.gate, r.flat};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &l = saved[0], &lse = saved[1], &flat = saved[2];
    c10::cuda::CUDAGuard guard(l.device());
    Tensor dl = at::empty(l.sizes(), l.options());
    Tensor dg = g[0].to(at::kFloat).contiguous();
    check(mcclMoeTokenBackward(nullptr, flat.data_ptr<int32_t>(), dg.data_ptr<float>(), l.data_ptr(), lse.data_ptr<float>(), nullptr,
                               dl.data_ptr(), nullptr, (int)l.size(0), (int)l.size(1), (int)ctx->saved_data["capacity"].toInt(), 0,
                               streamOf(l)), "mcclMoeTokenBackward");
    counters().moe++;
    return once({dl, Tensor()});
  }
};

bool routable(const Tensor& logits, int64_t capacity) {
  return !recorded() && ordinary(logits) && bf16Cuda(logits) && logits.dim() == 2 && logits.size(0) > 0 && logits.size(0) < (1 << 30) && logits.size(1) > 0 &&
         logits.size(1) <= mcclMoeRouteMaxExperts() && capacity > 0 && logits.size(1) * capacity <= INT32_MAX;
}

// (gate, flat) of top-1 routing, or None where the kernels do not cover the case.
py::object moeRoute(const Tensor& logits, int64_t capacity) {
  if (!routable(logits, capacity)) return py::none();
  variable_list r = RouteFn::apply(logits, capacity);
  return py::make_tuple(r[0], r[1]);
}

// Above this many experts the router's share of the token gradient is a matrix product of its own.
constexpr int64_t kFusedRouterExperts = 64;

struct MoeFn : torch::autograd::Function<MoeFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& xIn, const Tensor& router, const Tensor& wIn, const Tensor& wOut, int64_t capacity) {
    Below below;
    c10::cuda::CUDAGuard guard(xIn.device());
    Tensor x = xIn.contiguous();
    if (!aligned16(x)) x = x.clone();
    const int64_t T = x.size(0), d = x.size(1), E = router.size(0);
    mcclStream_t s = streamOf(x);
    Tensor logits = at::linear(x, router);
    Routed r = route(logits, capacity, true);
    Tensor slots = at::empty({E, capacity, d}, x.options());
    check(mcclMoeFillSlots(x.data_ptr(), r.inverse.data_ptr<int32_t>(), r.kept.data_ptr<int32_t>(), slots.data_ptr(), (int)E, (int)capacity,
                           (int)d, s), "mcclMoeFillSlots");
    Tensor pre = at::bmm(slots, wIn.transpose(1, 2));
    Tensor h = at::empty(pre.sizes(), pre.options());
    check(mcclSiluForward(pre.data_ptr(), h.data_ptr(), pre.numel(), s), "mcclSiluForward");
    Tensor out = at::bmm(h, wOut.transpose(1, 2));
    Tensor y = at::empty({T, d}, x.options());
    check(mcclMoeCombine(out.data_ptr(), r.flat.data_ptr<int32_t>(), r.gate.data_ptr<float>(), y.data_ptr(), (int)T, (int)d, s), "mcclMoeCombine");
    counters().moe += 3;
    ctx->save_for_backward({x, router, wIn, wOut, logits, r.gate, r.lse, r.flat, r.inverse, r.kept, slots, pre, h, out});
    ctx->saved_data["capacity"] = capacity;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto v = ctx->get_saved_variables();
    const Tensor &x = v[0], &router = v[1], &wIn = v[2], &wOut = v[3], &logits = v[4], &gate = v[5], &lse = v[6], &flat = v[7],
                 &inverse = v[8], &kept = v[9], &slots = v[10], &pre = v[11], &h = v[12], &out = v[13];
    if (at::GradMode::is_enabled()) {                                // to be differentiated again: from the inputs, by operators
      const int64_t E = router.size(0), C = ctx->saved_data["capacity"].toInt(), d = x.size(1);
      Tensor rows = (flat >= 0).nonzero().squeeze(1), slot = flat.index({rows}).to(at::kLong);
      Tensor p = at::softmax(at::linear(x, router).to(at::kFloat), -1), top = std::get<0>(p.max(-1)).to(x.scalar_type());
      Tensor in = at::zeros({E * C, d}, x.options()).index_put({slot}, x.index({rows})).view({E, C, d});
      Tensor o = at::bmm(at::silu(at::bmm(in, wIn.transpose(1, 2))), wOut.transpose(1, 2)).view({E * C, d});
      Tensor y = at::zeros_like(x).index_put({rows}, o.index({slot}) * top.index({rows}).unsqueeze(1));
      variable_list of, ret(5);
      for (int i = 0; i < 4; ++i) if (ctx->needs_input_grad(i)) of.push_back(v[i]);
      variable_list dv = torch::autograd::grad({y}, of, {g[0]}, std::nullopt, true);
      for (int i = 0, k = 0; i < 4; ++i) if (ctx->needs_input_grad(i)) ret[i] = dv[k++];
      return ret;
    }
    Below below;
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t T = x.size(0), d = x.size(1), E = router.size(0), C = ctx->saved_data["capacity"].toInt();
    mcclStream_t s = streamOf(x);
    Tensor dy = g[0].contiguous();
    if (!aligned16(dy)) dy = dy.clone();
    Tensor dout = at::empty(out.sizes(), out.options()), dgate = at::empty({T}, gate.options());
    check(mcclMoeCombineBackward(dy.data_ptr(), out.data_ptr(), inverse.data_ptr<int32_t>(), kept.data_ptr<int32_t>(), gate.data_ptr<float>(),
                                 dout.data_ptr(), dgate.data_ptr<float>(), (int)E, (int)C, (int)d, s), "mcclMoeCombineBackward");
    Tensor dh = at::bmm(dout, wOut);                                 // [E, C, f]
    Tensor dwOut = ctx->needs_input_grad(3) ? at::bmm(dout.transpose(1, 2), h) : Tensor();
    check(mcclSiluBackward(pre.data_ptr(), dh.data_ptr(), dh.data_ptr(), dh.numel(), s), "mcclSiluBackward");
    Tensor dwIn = ctx->needs_input_grad(2) ? at::bmm(dh.transpose(1, 2), slots) : Tensor();
    Tensor dslots = dout;                                            // its gradient has been used: the memory serves again
    at::bmm_out(dslots, dh, wIn);
    Tensor dlogits = at::empty(logits.sizes(), logits.options()), dx = at::empty(x.sizes(), x.options());
    const bool fused = E <= kFusedRouterExperts;
    check(mcclMoeTokenBackward(dslots.data_ptr(), flat.data_ptr<int32_t>(), dgate.data_ptr<float>(), logits.data_ptr(), lse.data_ptr<float>(),
                               fused ? router.data_ptr() : nullptr, dlogits.data_ptr(), dx.data_ptr(), (int)T, (int)E, (int)C, (int)d, s),
          "mcclMoeTokenBackward");
    counters().moe += 2;
    if (!fused) at::addmm_out(dx, dx, dlogits, router);
    Tensor dRouter = ctx->needs_input_grad(1) ? at::mm(dlogits.t(), x) : Tensor();
    return {dx, dRouter, dwIn, dwOut, Tensor()};
  }
};

// The layer's output, or None where the kernels do not cover the case.
py::object moeLayer(const Tensor& x, const Tensor& router, const Tensor& wIn, const Tensor& wOut, int64_t capacity) {
  if (recorded() || !ordinary(x) || !bf16Cuda(x) || x.dim() != 2 || x.size(0) == 0 || x.size(0) >= (1 << 30) || x.size(1) % 8 || router.dim() != 2 || router.size(1) != x.size(1) ||
      router.size(0) > mcclMoeRouteMaxExperts() || capacity <= 0 || router.size(0) * capacity > INT32_MAX) return py::none();
  for (const Tensor* w : {&router, &wIn, &wOut})
    if (!ordinary(*w) || !bf16Cuda(*w) || !w->is_contiguous() || !aligned16(*w)) return py::none();
  if (wIn.dim() != 3 || wIn.size(0) != router.size(0) || wIn.size(2) != x.size(1) || wOut.dim() != 3 || wOut.size(0) != router.size(0) ||
      wOut.size(1) != x.size(1) || wOut.size(2) != wIn.size(1)) return py::none();
  return py::cast(MoeFn::apply(x, router, wIn, wOut, capacity));
}

}  // namespace

void bindMoe(py::module_& m) {
  m.def("moe_route", &moeRoute);
  m.def("moe_layer", &moeLayer);
}

}  // namespace mccl_torch
