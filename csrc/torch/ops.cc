// LayerNorm, cross-entropy, optimizer and GEMM entry points of the torch binding.
#include "common.h"

namespace mccl_torch {
namespace {

// ---- LayerNorm ------------------------------------------------------------------------------------------------------
bool normSupported(const Tensor& x, const Tensor& w, const Tensor& b) {
  const int64_t d = x.dim() > 0 ? x.size(-1) : 0;
  return x.numel() > 0 && !recorded() && ordinary(x) && ordinary(w) && ordinary(b) && bf16Cuda(x) && bf16Cuda(w) && bf16Cuda(b) &&
         layerNormWidth(d) && w.numel() == d && b.numel() == d && w.is_contiguous() && b.is_contiguous() && aligned16(w) && aligned16(b);
}

struct LayerNormFn : torch::autograd::Function<LayerNormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
    const int64_t d = x.size(-1), rows = x.numel() / d;
    Tensor xc = x.contiguous();
    if (!aligned16(xc)) xc = xc.clone();
    Tensor y = at::empty(x.sizes(), xc.options());
    Tensor stats = at::empty({2, rows}, xc.options().dtype(at::kFloat));
    float* mean = stats.data_ptr<float>();
    c10::cuda::CUDAGuard guard(x.device());
    check(mcclLayerNormForward(xc.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), mean, mean + rows, rows, (int)d, (float)eps,
                               streamOf(xc)), "mcclLayerNormForward");
    counters().norm++;
    ctx->save_for_backward({xc, w, stats, b});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &stats = saved[2];
    const int64_t d = x.size(-1), rows = x.numel() / d;
    if (at::GradMode::is_enabled()) {                                // to be differentiated again: from the inputs, by operators
      Tensor xs = x.reshape({rows, d}), dy = g[0].reshape({rows, d});
      auto r = at::native_layer_norm_backward(dy, xs, {d}, stats.select(0, 0).unsqueeze(1), stats.select(0, 1).unsqueeze(1), w, saved[3],
                                              {true, true, true});
      return {std::get<0>(r).view(x.sizes()), std::get<1>(r), std::get<2>(r), Tensor()};
    }
    Tensor dx = at::empty(x.sizes(), x.options()), dw = at::empty({d}, w.options()), db = at::empty({d}, w.options());
    Tensor dy = g[0].contiguous();
    if (!aligned16(dy)) dy = dy.clone();
    Tensor partial = at::empty({(int64_t)mcclLayerNormPartials(rows) * 2 * d}, stats.options());
    const float* mean = stats.data_ptr<float>();
    c10::cuda::CUDAGuard guard(x.device());
    check(mcclLayerNormBackward(x.data_ptr(), dy.data_ptr(), w.data_ptr(), mean, mean + rows, dx.data_ptr(), dw.data_ptr(), db.data_ptr(),
                                partial.data_ptr<float>(), rows, (int)d, streamOf(x)), "mcclLayerNormBackward");
    counters().norm += 2;
    return {dx, dw, db, Tensor()};
  }
};

// y, or None where the kernels do not cover the case (the caller falls back to torch).
py::object layerNorm(const Tensor& x, const Tensor& w, const Tensor& b, double eps) {
  if (!normSupported(x, w, b)) return py::none();
  return py::cast(LayerNormFn::apply(x, w, b, eps));
}

// ---- cross-entropy --------------------------------------------------------------------------------------------------
struct CrossEntropyFn : torch::autograd::Function<CrossEntropyFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& targets, int64_t vocab) {
    const int64_t rows = logits.size(0);
    Tensor perRow = at::empty({2, rows}, logits.options().dtype(at::kFloat));
    Tensor mean = at::empty({}, perRow.options());
    float* loss = perRow.data_ptr<float>();
    c10::cuda::CUDAGuard guard(logits.device());
    check(mcclCrossEntropyMean(logits.data_ptr(), rows, logits.stride(0), (int)vocab, targets.data_ptr<int64_t>(), loss, loss + rows,
                               mean.data_ptr<float>(), nullptr, streamOf(logits)), "mcclCrossEntropyForward");
    counters().loss++;
    ctx->save_for_backward({logits, targets, perRow});
    ctx->saved_data["vocab"] = vocab;
    return mean;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    Tensor logits = saved[0];
    const Tensor &targets = saved[1], &perRow = saved[2];
    const int64_t rows = logits.size(0);
    Tensor go = g[0].scalar_type() == at::kFloat ? g[0] : g[0].to(at::kFloat);
    c10::cuda::CUDAGuard guard(logits.device());
    // The gradient overwrites the logits: nothing downstream of the output projection reads them again.
    check(mcclCrossEntropyBackward(logits.data_ptr(), rows, logits.stride(0), (int)ctx->saved_data["vocab"].toInt(), (int)logits.size(1),
                                   targets.data_ptr<int64_t>(), perRow.data_ptr<float>() + rows, go.data_ptr<float>(), streamOf(logits)),
          "mcclCrossEntropyBackward");
    counters().loss++;
    return {logits, Tensor(), Tensor()};
  }
};

// None where an argument is not what the kernels take (the caller says which).
py::object crossEntropy(const Tensor& logits, const Tensor& targets, std::optional<int64_t> vocab) {
  if (!bf16Cuda(logits) || logits.dim() != 2 || logits.stride(1) != 1 || targets.scalar_type() != at::kLong || !targets.is_contiguous() ||
      targets.numel() != logits.size(0) || (!targets.is_cuda() && !targets.is_pinned())) return py::none();
  return py::cast(CrossEntropyFn::apply(logits, targets, vocab ? *vocab : logits.size(1)));
}

// ---- optimizer ------------------------------------------------------------------------------------------------------
mcclStream_t pick(const Tensor& t, std::optional<int64_t> stream) {
  return stream ? reinterpret_cast<mcclStream_t>(*stream) : streamOf(t);
}

bool flat(const Tensor& t, at::ScalarType dt, int64_t n) { return t.scalar_type() == dt && t.numel() == n; }

// The library's status; -1 where an argument is not what the kernel takes (the caller says which).
int adamw(const Tensor& param, const Tensor& master, const Tensor& m, const Tensor& v, const Tensor& grad, double lr, double b1, double b2,
           double eps, double wd, double gradScale, int64_t step, bool zeroGrad, const std::optional<Tensor>& normSq, double maxNorm,
           std::optional<int64_t> stream, const std::optional<Tensor>& hyper) {
  const int64_t n = param.numel();
  if (!bf16Cuda(param) || !flat(grad, at::kBFloat16, n) || !flat(master, at::kFloat, n) || !flat(m, at::kFloat, n) || !flat(v, at::kFloat, n))
    return -1;
  const float* norm = normSq ? normSq->data_ptr<float>() : nullptr;
  mcclStream_t s = pick(param, stream);
  mcclResult_t rc;
  if (hyper) {
    if (!hyper->is_cuda() || hyper->scalar_type() != at::kFloat || hyper->numel() < 3) return -1;
    rc = mcclFusedAdamWDeviceHyper(param.data_ptr(), master.data_ptr<float>(), m.data_ptr<float>(), v.data_ptr<float>(), grad.data_ptr(),
                                   (uint64_t)n, hyper->data_ptr<float>(), (float)b1, (float)b2, (float)eps, (float)wd, (float)gradScale,
                                   zeroGrad, norm, (float)maxNorm, s);
  } else {
    rc = mcclFusedAdamW(param.data_ptr(), master.data_ptr<float>(), m.data_ptr<float>(), v.data_ptr<float>(), grad.data_ptr(), (uint64_t)n,
                        (float)lr, (float)b1, (float)b2, (float)eps, (float)wd, (float)gradScale, (int)step, zeroGrad, norm, (float)maxNorm, s);
  }
  if (rc == mcclSuccess) counters().optim++;
  return rc;
}

int sumSquares(const Tensor& x, const Tensor& out, const Tensor& scratch, bool accumulate, std::optional<int64_t> stream) {
  if (!bf16Cuda(x) || out.scalar_type() != at::kFloat || scratch.scalar_type() != at::kFloat) return -1;
  const mcclResult_t rc = mcclSumSquaresBf16(x.data_ptr(), (uint64_t)x.numel(), scratch.data_ptr<float>(), (uint64_t)scratch.numel(),
                                             out.data_ptr<float>(), accumulate, pick(x, stream));
  if (rc == mcclSuccess) counters().optim++;
  return rc;
}

// ---- GEMM -----------------------------------------------------------------------------------------------------------
// out = act(x w^T); the library's status where it failed; None where a shape or type is not what the kernels take (the caller says which).
py::object gemm(const Tensor& x, const Tensor& w, const std::optional<Tensor>& out, int64_t epilogue, int64_t maxCtas,
                std::optional<int64_t> stream, std::optional<bool> twoSm) {
  if (!bf16Cuda(x) || !bf16Cuda(w) || x.dim() != 2 || w.dim() != 2 || !x.is_contiguous() || !w.is_contiguous()) return py::none();
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  if (w.size(1) != K || M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 64 || K % 64) return py::none();
  const bool two = twoSm ? *twoSm : M % 256 == 0;
  if (two && M % 256) return py::none();
  Tensor y = out ? *out : at::empty({M, N}, x.options());
  auto* fn = two ? mcclTpGemm2 : mcclTpGemm;
  const mcclResult_t rc = fn(x.data_ptr(), w.data_ptr(), y.data_ptr(), (int)M, (int)N, (int)K, (int)epilogue, (int)maxCtas, pick(x, stream));
  if (rc != mcclSuccess) return py::cast((int)rc);
  counters().gemm++;
  return py::cast(y);
}

// ---- SiLU MLP on one rank ---------------------------------------------------------------------------------------------
// y = silu(x w_up^T) w_down^T.  The up product stores its sums beside the activation, so the backward pass is four products
// and one elementwise pass; without gradients they are not kept.
struct MlpFn : torch::autograd::Function<MlpFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& xIn, const Tensor& wUp, const Tensor& wDown, bool keep) {
    Below below;
    c10::cuda::CUDAGuard guard(xIn.device());
    Tensor x = xIn.contiguous();
    const int T = (int)x.size(0), h = (int)x.size(1), f = (int)wUp.size(0);
    Tensor act = at::empty({T, f}, x.options()), pre = keep ? at::empty({T, f}, x.options()) : Tensor(), y = at::empty({T, h}, x.options());
    check(mcclTpGemmKeepPre(x.data_ptr(), wUp.data_ptr(), act.data_ptr(), keep ? pre.data_ptr() : nullptr, T, f, h, MCCL_EPILOGUE_SILU, streamOf(x)),
          "mcclTpGemmKeepPre");
    check(mcclTpGemmKeepPre(act.data_ptr(), wDown.data_ptr(), y.data_ptr(), nullptr, T, h, f, MCCL_EPILOGUE_NONE, streamOf(x)), "mcclTpGemmKeepPre");
    counters().gemm += 2;
    if (keep) ctx->save_for_backward({x, wUp, wDown, act, pre});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto v = ctx->get_saved_variables();
    const Tensor &x = v[0], &wUp = v[1], &wDown = v[2], &act = v[3], &pre = v[4];
    if (at::GradMode::is_enabled()) {                                // to be differentiated again: from the inputs, by operators
      variable_list in;
      for (int i = 0; i < 3; ++i) if (ctx->needs_input_grad(i)) in.push_back(v[i]);
      Tensor y = at::linear(at::silu(at::linear(x, wUp)), wDown);
      variable_list d = torch::autograd::grad({y}, in, {g[0]}, std::nullopt, true), ret(4);
      for (int i = 0, k = 0; i < 3; ++i) if (ctx->needs_input_grad(i)) ret[i] = d[k++];
      return ret;
    }
    Below below;
    c10::cuda::CUDAGuard guard(x.device());
    Tensor dy = g[0].contiguous();
    variable_list ret(4);
    if (ctx->needs_input_grad(2)) ret[2] = at::mm(dy.t(), act);
    Tensor du = at::mm(dy, wDown);
    check(mcclSiluBackward(pre.data_ptr(), du.data_ptr(), du.data_ptr(), du.numel(), streamOf(x)), "mcclSiluBackward");
    if (ctx->needs_input_grad(1)) ret[1] = at::mm(du.t(), x);
    if (ctx->needs_input_grad(0)) ret[0] = at::mm(du, wUp);
    return ret;
  }
};

// None where the kernels do not cover the case.
py::object mlp(const Tensor& x, const Tensor& wUp, const Tensor& wDown) {
  if (recorded()) return py::none();
  for (const Tensor* t : {&x, &wUp, &wDown})
    if (!ordinary(*t) || !bf16Cuda(*t) || t->dim() != 2 || !aligned16(*t)) return py::none();
  const int64_t T = x.size(0), h = x.size(1), f = wUp.size(0);
  if (!wUp.is_contiguous() || !wDown.is_contiguous() || wUp.size(1) != h || wDown.size(0) != h || wDown.size(1) != f || T <= 0 || T % 128 || h % 64 ||
      f % 64) return py::none();
  const bool keep = at::GradMode::is_enabled() && (x.requires_grad() || wUp.requires_grad() || wDown.requires_grad());
  return py::cast(MlpFn::apply(x, wUp, wDown, keep));
}

// (silu(u), du) from the pre-activation and the gradient of the activation.
std::pair<Tensor, Tensor> siluBoth(const Tensor& u, const Tensor& dh) {
  TORCH_CHECK(bf16Cuda(u) && bf16Cuda(dh) && u.is_contiguous() && dh.is_contiguous() && u.numel() == dh.numel(), "silu_both: bf16 cuda tensors");
  Tensor h = at::empty_like(u), du = at::empty_like(u);
  check(mcclSiluForwardBackward(u.data_ptr(), dh.data_ptr(), h.data_ptr(), du.data_ptr(), u.numel(), streamOf(u)), "mcclSiluForwardBackward");
  return {h, du};
}

// Tanh-GELU and, with a gradient, the gradient of x and its column sums.
Tensor geluForward(const Tensor& x) {
  TORCH_CHECK(bf16Cuda(x) && x.is_contiguous(), "gelu: a contiguous bf16 cuda tensor");
  Tensor y = at::empty_like(x);
  check(mcclGeluForward(x.data_ptr(), y.data_ptr(), x.numel(), streamOf(x)), "mcclGeluForward");
  return y;
}
std::pair<Tensor, Tensor> geluBackward(const Tensor& x, const Tensor& dy) {
  TORCH_CHECK(bf16Cuda(x) && bf16Cuda(dy) && x.dim() == 2 && x.is_contiguous() && dy.is_contiguous() && x.sizes() == dy.sizes(), "gelu: bf16 cuda matrices");
  Tensor dx = at::empty_like(x), db = at::empty({x.size(1)}, x.options());
  Tensor scratch = at::empty({mcclColumnSumScratch(x.size(0), (int)x.size(1), 1)}, x.options().dtype(at::kFloat));
  check(mcclGeluBackward(x.data_ptr(), dy.data_ptr(), dx.data_ptr(), db.data_ptr(), 0, scratch.data_ptr<float>(), x.size(0), (int)x.size(1),
                         streamOf(x)), "mcclGeluBackward");
  return {dx, db};
}

}  // namespace

void bindOps(py::module_& m) {
  m.def("layer_norm", &layerNorm);
  m.def("cross_entropy", &crossEntropy);
  m.def("adamw", &adamw);
  m.def("sum_squares", &sumSquares);
  m.def("gemm", &gemm);
  m.def("mlp", &mlp);
  m.def("silu_both", &siluBoth);
  m.def("gelu_forward", &geluForward);
  m.def("gelu_backward", &geluBackward);
  m.def("launches", [](const std::string& what) -> int64_t {
    Counters& c = counters();
    if (what == "norm") return c.norm;
    if (what == "loss") return c.loss;
    if (what == "optim") return c.optim;
    if (what == "gemm") return c.gemm;
    return c.moe;
  });
}

}  // namespace mccl_torch

PYBIND11_MODULE(mccl_torch, m) {
  mccl_torch::bindOps(m);
  mccl_torch::bindComm(m);
  mccl_torch::bindMoe(m);
  mccl_torch::bindGpt2(m);
  mccl_torch::bindLlama(m);
}
