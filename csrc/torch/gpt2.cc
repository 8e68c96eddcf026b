// The GPT-2 style decoder's nodes: embedding, the two halves of a block around attention, the final norm and the loss head.
//
// A block as separate tensor operations runs about 15 launches forward and 35 backward, a third of them passes that only add
// (residuals, gradients into their buckets) or only sum (bias gradients).  Here
//   * the residual add is done by the norm behind it: a block hands on its residual stream and its MLP output un-added;
//   * the column sums of a gradient (a bias gradient) fall out of the kernel that writes the gradient: the norm's backward
//     kernel for the projections that feed a residual add, the GELU's for the up projection;
//   * weight gradients are accumulated by the matrix product itself (gradsink.h).
// The bias of a projection whose output is added by the NEXT node gets its gradient there; it is passed along for that.
#include "nodes.h"

namespace mccl_torch {
namespace {

// Three adjacent matrices (or vectors) of one storage as one, in memory order; undefined where they are not adjacent.
Tensor adjacent(const Tensor& a, const Tensor& b, const Tensor& c) {
  const char *pa = (const char*)a.data_ptr(), *pb = (const char*)b.data_ptr(), *pc = (const char*)c.data_ptr();
  const int64_t bytes = a.numel() * a.element_size();
  if (pb != pa + bytes || pc != pb + bytes || !a.storage().is_alias_of(b.storage()) || !a.storage().is_alias_of(c.storage())) return Tensor();
  auto sizes = a.sizes().vec();
  sizes[0] *= 3;
  return a.dim() == 2 ? a.as_strided(sizes, {sizes[1], 1}) : a.as_strided(sizes, {1});
}

// sum = x + pending (pending may be missing: sum = x) and its norm.  `exact`: at widths this library had no kernel for, a
// forward pass without gradients keeps the tensor library's norm, bit for bit (a last-bit difference in the first norm is a
// difference of a percent in the logits of a 12-layer model in bf16, so scores would not compare with recorded ones).
void addNorm(const Tensor& x, const Tensor* pending, const Tensor& lw, const Tensor& lb, double eps, bool exact, Tensor* sum, Tensor* h, Tensor* stats) {
  const int64_t T = x.size(0), d = x.size(1);
  if (exact && d != 256 && d != 512 && d != 1024) {
    *sum = pending ? at::add(x, *pending) : at::alias(x);
    *h = std::get<0>(at::native_layer_norm(*sum, {d}, lw, lb, eps));
    return;
  }
  Norm n = normStats(x, T);
  *stats = n.stats;
  *h = at::empty({T, d}, x.options());
  if (pending) {
    *sum = at::empty({T, d}, x.options());
    check(mcclAddLayerNormForward(x.data_ptr(), pending->data_ptr(), lw.data_ptr(), lb.data_ptr(), sum->data_ptr(), h->data_ptr(), n.mean(),
                                  n.rstd(T), T, (int)d, (float)eps, streamOf(x)), "mcclAddLayerNormForward");
  } else {
    *sum = at::alias(x);
    check(mcclLayerNormForward(x.data_ptr(), lw.data_ptr(), lb.data_ptr(), h->data_ptr(), n.mean(), n.rstd(T), T, (int)d, (float)eps,
                               streamOf(x)), "mcclLayerNormForward");
  }
  counters().norm++;
}

// ---- first half: (residual, pending) -> residual sum, norm, q, k, v -----------------------------------------------------
struct BlockInFn : torch::autograd::Function<BlockInFn> {
  // Outputs: residual [T, d], q, k, v [b, h, s, hd].
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& pending, const OptTensor& pendingBias, const Tensor& lw,
                               const Tensor& lb, const Tensor& wq, const Tensor& bq, const Tensor& wk, const Tensor& bk, const Tensor& wv,
                               const Tensor& bv, int64_t b, int64_t s, int64_t heads, double eps, bool sink, bool exact) {
    Below below;
    const int64_t T = x.size(0), d = x.size(1), hd = d / heads;
    Tensor sum, h, stats;
    addNorm(x, pending ? &*pending : nullptr, lw, lb, eps, exact, &sum, &h, &stats);
    auto split = [&](const Tensor& t, int64_t rowStride, int64_t offset) {
      return t.as_strided({b, heads, s, hd}, {s * rowStride, hd, rowStride, 1}, t.storage_offset() + offset);
    };
    Tensor q, k, v;
    // One product for the three projections where their weights lie next to each other (a bucket keeps parameters in
    // reverse order of registration: v, k, q).
    Tensor w3 = adjacent(wv, wk, wq), b3 = w3.defined() ? adjacent(bv, bk, bq) : Tensor();
    if (b3.defined()) {
      Tensor o = at::linear(h, w3, b3);
      v = split(o, 3 * d, 0); k = split(o, 3 * d, d); q = split(o, 3 * d, 2 * d);
    } else {
      q = split(at::linear(h, wq, bq), d, 0);
      k = split(at::linear(h, wk, bk), d, 0);
      v = split(at::linear(h, wv, bv), d, 0);
    }
    // Without a pending term the sum is the input: saved as such, so that a change made to it in place is noticed.
    ctx->save_for_backward({pending ? sum : x, h, stats, lw, lb, wq, bq, wk, bk, wv, bv, pendingBias ? *pendingBias : Tensor()});
    ctx->saved_data["sink"] = sink;
    ctx->saved_data["pending"] = pending.has_value();
    return {sum, q, k, v};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &sum = saved[0], &h = saved[1], &stats = saved[2], &lw = saved[3], &lb = saved[4], &wq = saved[5], &bq = saved[6],
                 &wk = saved[7], &bk = saved[8], &wv = saved[9], &bv = saved[10], &pb = saved[11];
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const bool pending = ctx->saved_data["pending"].toBool();
    const int64_t T = h.size(0), d = h.size(1);
    mcclStream_t s = streamOf(h);
    auto zeros = [&] { return at::zeros({T, d}, h.options()); };
    Tensor dq = g[1].defined() ? fromHeads(g[1], T, d) : zeros(), dk = g[2].defined() ? fromHeads(g[2], T, d) : zeros(),
           dv = g[3].defined() ? fromHeads(g[3], T, d) : zeros();
    Tensor dwq, dwk, dwv, dhv, dhk, dhq;
    VectorGrads db(sink, {&bv, &bk, &bq});
    Tensor scratch = columnScratch(h, T, d, 3);
    const void* in[3] = {dv.data_ptr(), dk.data_ptr(), dq.data_ptr()};
    void* out[3] = {db.t[0].data_ptr(), db.t[1].data_ptr(), db.t[2].data_ptr()};
    Tensor w3 = adjacent(wv, wk, wq);
    if (w3.defined()) {
      // The weights as one matrix: the gradients are laid side by side on the pass that sums their columns, and one product
      // gives the norm's gradient, another the three weight gradients where those are one matrix too.
      Tensor d3 = at::empty({T, 3 * d}, h.options());
      check(mcclPackColumnSums(in, d3.data_ptr(), out, 3, db.direct, scratch.data_ptr<float>(), T, (int)d, s), "mcclPackColumnSums");
      dhv = at::mm(d3, w3);
      Tensor gv = sink.buffer(wv), gk = sink.buffer(wk), gq = sink.buffer(wq);
      Tensor g3 = gv.defined() && gk.defined() && gq.defined() ? adjacent(gv, gk, gq) : Tensor();
      if (g3.defined()) {
        at::addmm_out(g3, g3, d3.t(), h);
      } else {
        weightGrad(sink, wv, dv, h, &dwv);
        weightGrad(sink, wk, dk, h, &dwk);
        weightGrad(sink, wq, dq, h, &dwq);
      }
    } else {
      check(mcclColumnSums(in, out, 3, db.direct, scratch.data_ptr<float>(), T, (int)d, d, s), "mcclColumnSums");
      dhv = at::mm(dv, wv); dhk = at::mm(dk, wk); dhq = at::mm(dq, wq);      // the norm's backward kernel adds them up
      weightGrad(sink, wv, dv, h, &dwv);
      weightGrad(sink, wk, dk, h, &dwk);
      weightGrad(sink, wq, dq, h, &dwq);
    }
    const void *part2 = dhk.defined() ? dhk.data_ptr() : nullptr, *part3 = dhq.defined() ? dhq.data_ptr() : nullptr;
    Tensor dx = at::empty({T, d}, h.options());
    Tensor partial = at::empty({(int64_t)mcclLayerNormPartials(T) * 3 * d}, stats.options());
    const float* mean = stats.data_ptr<float>();
    variable_list ret(17);
    if (g[0].defined()) {
      Tensor dres = rows2d(g[0], T, d);
      if (pb.defined()) {
        VectorGrads dn(sink, {&lw, &lb, &pb});
        check(mcclAddLayerNormBackward(sum.data_ptr(), dhv.data_ptr(), part2, part3, dres.data_ptr(), lw.data_ptr(), mean, mean + T, dx.data_ptr(),
                                       dn.t[0].data_ptr(), dn.t[1].data_ptr(), dn.t[2].data_ptr(), dn.direct, partial.data_ptr<float>(), T,
                                       (int)d, s), "mcclAddLayerNormBackward");
        ret[3] = dn.ret(0); ret[4] = dn.ret(1); ret[2] = dn.ret(2);
      } else {
        VectorGrads dn(sink, {&lw, &lb});
        check(mcclAddLayerNormBackward(sum.data_ptr(), dhv.data_ptr(), part2, part3, dres.data_ptr(), lw.data_ptr(), mean, mean + T, dx.data_ptr(),
                                       dn.t[0].data_ptr(), dn.t[1].data_ptr(), nullptr, dn.direct, partial.data_ptr<float>(), T, (int)d, s),
              "mcclAddLayerNormBackward");
        ret[3] = dn.ret(0); ret[4] = dn.ret(1);
      }
    } else {                                       // nobody uses the residual: the plain norm, and the bias on its own
      ret[3] = at::empty(lw.sizes(), lw.options());
      ret[4] = at::empty(lb.sizes(), lb.options());
      Tensor dh = part2 ? dhv.add_(dhk).add_(dhq) : dhv;
      check(mcclLayerNormBackward(sum.data_ptr(), dh.data_ptr(), lw.data_ptr(), mean, mean + T, dx.data_ptr(), ret[3].data_ptr(),
                                  ret[4].data_ptr(), partial.data_ptr<float>(), T, (int)d, s), "mcclLayerNormBackward");
      if (pb.defined()) ret[2] = dx.sum(0);
    }
    counters().norm += 2;
    ret[0] = dx;
    if (pending) ret[1] = dx;
    ret[5] = dwq; ret[6] = db.ret(2); ret[7] = dwk; ret[8] = db.ret(1); ret[9] = dwv; ret[10] = db.ret(0);
    return once(std::move(ret));
  }
};

// ---- second half: attention output and residual -> residual sum, MLP output ---------------------------------------------
struct BlockOutFn : torch::autograd::Function<BlockOutFn> {
  // Outputs: residual after attention [T, d], MLP output (with its bias) [T, d].  outBiasHere: the bias gradient of the down
  // projection is taken by this node and not by the one that adds its output.
  static variable_list forward(AutogradContext* ctx, const Tensor& a, const Tensor& res, const Tensor& wo, const Tensor& bo, const Tensor& lw,
                               const Tensor& lb, const Tensor& wf, const Tensor& bf, const Tensor& wd, const Tensor& bd, bool outBiasHere,
                               double eps, bool sink, bool exact) {
    Below below;
    const int64_t T = res.size(0), d = res.size(1);
    mcclStream_t s = streamOf(res);
    Tensor a2 = fromHeads(a, T, d);
    Tensor p = at::linear(a2, wo, bo);
    Tensor x1, h, stats;
    addNorm(res, &p, lw, lb, eps, exact, &x1, &h, &stats);
    Tensor u = at::linear(h, wf, bf);
    Tensor act = at::empty(u.sizes(), u.options());
    check(mcclGeluForward(u.data_ptr(), act.data_ptr(), u.numel(), s), "mcclGeluForward");
    Tensor y = at::linear(act, wd, bd);
    ctx->save_for_backward({a2, x1, h, stats, u, act, wo, bo, lw, lb, wf, bf, wd, bd});
    ctx->saved_data["sink"] = sink;
    ctx->saved_data["bias"] = outBiasHere;
    ctx->saved_data["b"] = a.size(0);
    ctx->saved_data["h"] = a.size(1);
    return {x1, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &a2 = saved[0], &x1 = saved[1], &h = saved[2], &stats = saved[3], &u = saved[4], &act = saved[5], &wo = saved[6],
                 &bo = saved[7], &lw = saved[8], &lb = saved[9], &wf = saved[10], &bf = saved[11], &wd = saved[12], &bd = saved[13];
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = h.size(0), d = h.size(1), f = u.size(1), b = ctx->saved_data["b"].toInt(), heads = ctx->saved_data["h"].toInt();
    mcclStream_t s = streamOf(h);
    variable_list ret(14);
    Tensor dy = g[1].defined() ? rows2d(g[1], T, d) : at::zeros({T, d}, h.options());
    Tensor dres = g[0].defined() ? rows2d(g[0], T, d) : at::zeros({T, d}, h.options());
    if (ctx->saved_data["bias"].toBool()) {
      VectorGrads db(sink, {&bd});
      Tensor scratch = columnScratch(h, T, d, 1);
      const void* in[1] = {dy.data_ptr()};
      void* out[1] = {db.t[0].data_ptr()};
      check(mcclColumnSums(in, out, 1, db.direct, scratch.data_ptr<float>(), T, (int)d, d, s), "mcclColumnSums");
      ret[9] = db.ret(0);
    }
    Tensor du = at::mm(dy, wd);
    weightGrad(sink, wd, dy, act, &ret[8]);
    {
      VectorGrads db(sink, {&bf});
      Tensor scratch = columnScratch(h, T, f, 1);
      check(mcclGeluBackward(u.data_ptr(), du.data_ptr(), du.data_ptr(), db.t[0].data_ptr(), db.direct, scratch.data_ptr<float>(), T, (int)f, s),
            "mcclGeluBackward");
      ret[7] = db.ret(0);
    }
    Tensor dh = at::mm(du, wf);
    weightGrad(sink, wf, du, h, &ret[6]);
    Tensor dx = at::empty({T, d}, h.options());
    {
      VectorGrads dn(sink, {&lw, &lb, &bo});
      Tensor partial = at::empty({(int64_t)mcclLayerNormPartials(T) * 3 * d}, stats.options());
      const float* mean = stats.data_ptr<float>();
      check(mcclAddLayerNormBackward(x1.data_ptr(), dh.data_ptr(), nullptr, nullptr, dres.data_ptr(), lw.data_ptr(), mean, mean + T, dx.data_ptr(),
                                     dn.t[0].data_ptr(), dn.t[1].data_ptr(), dn.t[2].data_ptr(), dn.direct, partial.data_ptr<float>(), T, (int)d,
                                     s), "mcclAddLayerNormBackward");
      counters().norm += 2;
      ret[4] = dn.ret(0); ret[5] = dn.ret(1); ret[3] = dn.ret(2);
    }
    Tensor da = at::mm(dx, wo);
    weightGrad(sink, wo, dx, a2, &ret[2]);
    ret[0] = da.view({b, T / b, heads, d / heads}).transpose(1, 2);
    ret[1] = dx;
    return once(std::move(ret));
  }
};

// ---- final norm of (residual, pending) --------------------------------------------------------------------------------
struct FinalNormFn : torch::autograd::Function<FinalNormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& pending, const OptTensor& pendingBias, const Tensor& lw,
                        const Tensor& lb, double eps, bool sink, bool exact) {
    Below below;
    Tensor sum, h, stats;
    addNorm(x, &pending, lw, lb, eps, exact, &sum, &h, &stats);
    ctx->save_for_backward({sum, stats, lw, lb, pendingBias ? *pendingBias : Tensor()});
    ctx->saved_data["sink"] = sink;
    return h;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &sum = saved[0], &stats = saved[1], &lw = saved[2], &lb = saved[3], &pb = saved[4];
    Below below;
    c10::cuda::CUDAGuard guard(sum.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = sum.size(0), d = sum.size(1);
    mcclStream_t s = streamOf(sum);
    Tensor dh = rows2d(g[0], T, d), dx = at::empty({T, d}, sum.options());
    Tensor partial = at::empty({(int64_t)mcclLayerNormPartials(T) * 2 * d}, stats.options());
    const float* mean = stats.data_ptr<float>();
    variable_list ret(8);
    VectorGrads dn(sink, {&lw, &lb});
    check(mcclAddLayerNormBackward(sum.data_ptr(), dh.data_ptr(), nullptr, nullptr, nullptr, lw.data_ptr(), mean, mean + T, dx.data_ptr(), dn.t[0].data_ptr(),
                                   dn.t[1].data_ptr(), nullptr, dn.direct, partial.data_ptr<float>(), T, (int)d, s), "mcclAddLayerNormBackward");
    counters().norm += 2;
    ret[3] = dn.ret(0); ret[4] = dn.ret(1);
    if (pb.defined()) {
      VectorGrads db(sink, {&pb});
      Tensor scratch = columnScratch(sum, T, d, 1);
      const void* in[1] = {dx.data_ptr()};
      void* out[1] = {db.t[0].data_ptr()};
      check(mcclColumnSums(in, out, 1, db.direct, scratch.data_ptr<float>(), T, (int)d, d, s), "mcclColumnSums");
      ret[2] = db.ret(0);
    }
    ret[0] = dx;
    ret[1] = dx;
    return once(std::move(ret));
  }
};

// ---- embedding ----------------------------------------------------------------------------------------------------------
struct EmbedFn : torch::autograd::Function<EmbedFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& idx, const Tensor& table, const OptTensor& pos, bool sink) {
    Below below;
    const int64_t T = idx.numel(), d = table.size(1), seq = idx.size(-1);
    Tensor i = idx.contiguous(), out = at::empty({T, d}, table.options());
    check(mcclEmbeddingForward(i.data_ptr<int64_t>(), table.data_ptr(), pos ? pos->data_ptr() : nullptr, out.data_ptr(), T, (int)seq,
                               table.size(0), (int)d,
                               streamOf(out)), "mcclEmbeddingForward");
    ctx->save_for_backward({i, table, pos ? *pos : Tensor()});
    ctx->saved_data["sink"] = sink;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &idx = saved[0], &table = saved[1], &pos = saved[2];
    Below below;
    c10::cuda::CUDAGuard guard(table.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = idx.numel(), d = table.size(1), seq = idx.size(-1), V = table.size(0);
    Tensor dy = rows2d(g[0], T, d);
    variable_list ret(4);
    const bool here = T <= mcclEmbeddingMaxTokens();
    const bool withPos = pos.defined();
    Tensor dt = here ? sink.buffer(table) : Tensor(), dp = here && withPos ? sink.buffer(pos) : Tensor();
    const bool direct = dt.defined() && (dp.defined() || !withPos);
    if (!direct) {
      if (here) {
        ret[1] = dt = at::zeros(table.sizes(), table.options());
        if (withPos) ret[2] = dp = at::zeros(pos.sizes(), pos.options());
      } else {
        // Too many tokens for the kernel's scan: the sorting form of the tensor library.
        ret[1] = at::embedding_dense_backward(dy, idx.view({T}), V, -1, false);
        if (withPos) {
          ret[2] = at::zeros(pos.sizes(), pos.options());
          ret[2].narrow(0, 0, seq).copy_(dy.view({T / seq, seq, d}).sum(0));
        }
        return once(std::move(ret));
      }
    }
    Tensor count = at::empty({V}, idx.options().dtype(at::kInt));
    check(mcclEmbeddingBackward(idx.data_ptr<int64_t>(), dy.data_ptr(), dt.data_ptr(), withPos ? dp.data_ptr() : nullptr, count.data_ptr<int32_t>(), T, (int)seq, V,
                                (int)d, streamOf(dy)), "mcclEmbeddingBackward");
    return once(std::move(ret));
  }
};

// ---- head: projection and cross-entropy ----------------------------------------------------------------------------
struct HeadLossFn : torch::autograd::Function<HeadLossFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& h, const Tensor& w, const Tensor& targets, int64_t vocab, bool meanOfUsed,
                        bool sink) {
    Below below;
    const int64_t T = h.size(0);
    Tensor logits = at::linear(h, w);
    Tensor t = targets.contiguous();
    Tensor perRow = at::empty({2 * T + 1}, h.options().dtype(at::kFloat)), mean = at::empty({}, perRow.options());
    float* loss = perRow.data_ptr<float>();
    check(mcclCrossEntropyMean(logits.data_ptr(), T, logits.stride(0), (int)vocab, t.data_ptr<int64_t>(), loss, loss + T, mean.data_ptr<float>(),
                               meanOfUsed ? loss + 2 * T : nullptr, streamOf(h)), "mcclCrossEntropyForward");
    counters().loss++;
    ctx->save_for_backward({h, w, t, logits, perRow});
    ctx->saved_data["vocab"] = vocab;
    ctx->saved_data["used"] = meanOfUsed;
    ctx->saved_data["sink"] = sink;
    return mean;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &h = saved[0], &w = saved[1], &t = saved[2], &perRow = saved[4];
    Tensor logits = saved[3];
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = h.size(0);
    Tensor go = g[0].scalar_type() == at::kFloat ? g[0] : g[0].to(at::kFloat);
    float* rows = perRow.data_ptr<float>();
    check(mcclCrossEntropyMeanBackward(logits.data_ptr(), T, logits.stride(0), (int)ctx->saved_data["vocab"].toInt(), (int)logits.size(1),
                                       t.data_ptr<int64_t>(), rows + T, go.data_ptr<float>(),
                                       ctx->saved_data["used"].toBool() ? rows + 2 * T : nullptr, streamOf(h)),
          "mcclCrossEntropyBackward");
    counters().loss++;
    variable_list ret(6);
    ret[0] = at::mm(logits, w);
    weightGrad(sink, w, logits, h, &ret[1]);
    return once(std::move(ret));
  }
};

// ---- entry points ---------------------------------------------------------------------------------------------------------
// One block on x + pending (both [T, d]; pending may be missing).  params: ln1 w b, q w b, k w b, v w b, proj w b, ln2 w b,
// fc w b, out w b.  Returns (residual, MLP output), whose sum is the block's output, or None where the kernels do not cover
// the case.
py::object block(const Tensor& x, const OptTensor& pending, const OptTensor& pendingBias, const std::vector<Tensor>& p, int64_t b, int64_t s,
                 int64_t heads, bool outBiasHere, double eps, bool sink) {
  if (p.size() != 16 || x.dim() != 2 || !usable(x, p) || !attentionOnce()) return py::none();
  const int64_t d = x.size(1), f = p[12].size(0);
  if (heads <= 0 || d % heads || (d / heads) % 8 || f % 8 || x.size(0) != b * s) return py::none();
  if (pending && (!plainBf16(*pending, x) || !shaped(*pending, x.sizes()))) return py::none();
  if (pendingBias && (!plainBf16(*pendingBias, x) || !shaped(*pendingBias, {d}))) return py::none();
  for (int i : {0, 1, 3, 5, 7, 9, 10, 11, 15}) if (!shaped(p[i], {d})) return py::none();
  for (int i : {2, 4, 6, 8}) if (!shaped(p[i], {d, d})) return py::none();
  if (!shaped(p[12], {f, d}) || !shaped(p[13], {f}) || !shaped(p[14], {d, f})) return py::none();
  c10::cuda::CUDAGuard guard(x.device());
  const bool exact = !at::GradMode::is_enabled();
  variable_list in = BlockInFn::apply(x, pending, pendingBias, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], b, s, heads, eps, sink, exact);
  Tensor a = at::scaled_dot_product_attention(in[1], in[2], in[3], {}, 0.0, true);
  variable_list out = BlockOutFn::apply(a, in[0], p[8], p[9], p[10], p[11], p[12], p[13], p[14], p[15], outBiasHere, eps, sink, exact);
  return py::make_tuple(out[0], out[1]);
}

// table[idx] + pos (pos may be missing) as [tokens, d].
py::object embed(const Tensor& idx, const Tensor& table, const OptTensor& pos, bool sink) {
  if (!ordinary(idx) || idx.device() != table.device() || idx.dim() == 0 || idx.scalar_type() != at::kLong || idx.numel() == 0 ||
      !usable(table, {table}) || table.dim() != 2) return py::none();
  if (pos && (!plainBf16(*pos, table) || pos->dim() != 2 || pos->size(1) != table.size(1) || idx.size(-1) > pos->size(0))) return py::none();
  c10::cuda::CUDAGuard guard(table.device());
  return py::cast(EmbedFn::apply(idx, table, pos, sink));
}

py::object finalNorm(const Tensor& x, const Tensor& pending, const OptTensor& pendingBias, const Tensor& w, const Tensor& b, double eps, bool sink) {
  if (!usable(x, {pending, w, b}) || x.dim() != 2 || !shaped(pending, x.sizes()) || !shaped(w, {x.size(1)}) || !shaped(b, {x.size(1)}))
    return py::none();
  if (pendingBias && (!plainBf16(*pendingBias, x) || !shaped(*pendingBias, {x.size(1)}))) return py::none();
  c10::cuda::CUDAGuard guard(x.device());
  return py::cast(FinalNormFn::apply(x, pending, pendingBias, w, b, eps, sink, !at::GradMode::is_enabled()));
}

// Mean cross-entropy of h w^T: over all rows, or over those whose target is a column (`meanOfUsed`).
py::object headLoss(const Tensor& h, const Tensor& w, const Tensor& targets, int64_t vocab, bool meanOfUsed, bool sink) {
  if (!usable(h, {w}) || h.dim() != 2 || w.dim() != 2 || w.size(1) != h.size(1) || !ordinary(targets) || targets.device() != h.device() || targets.scalar_type() != at::kLong || targets.numel() != h.size(0) || w.size(0) < vocab) return py::none();
  c10::cuda::CUDAGuard guard(h.device());
  return py::cast(HeadLossFn::apply(h, w, targets.reshape({-1}), vocab, meanOfUsed, sink));
}

}  // namespace

void bindGpt2(py::module_& m) {
  m.def("gpt2_block", &block);
  m.def("decoder_embed", &embed);
  m.def("gpt2_final_norm", &finalNorm);
  m.def("decoder_head_loss", &headLoss);
}

}  // namespace mccl_torch
