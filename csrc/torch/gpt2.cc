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

// The norms here give FusedLayerNorm's results: the library's kernel at the widths it has one for, the tensor library's
// elsewhere.  A model then scores and trains with the same bits on this route and on the plain one.  (Another order of a
// norm's sums is a last bit of some of its results; in bf16, twelve layers on, that is a percent of the logits, and over 24
// layers and two steps of training up to 0.03 of the moments, more than two runs of one route lie apart.)
struct Norm { Tensor sum, h, mean, rstd; };        // own kernels: both statistics in `mean`, rstd undefined

Norm addNorm(const Tensor& x, const Tensor* pending, const Tensor& lw, const Tensor& lb, double eps) {
  const int64_t T = x.size(0), d = x.size(1);
  Norm n;
  if (!layerNormWidth(d)) {
    n.sum = pending ? at::add(x, *pending) : at::alias(x);
    std::tie(n.h, n.mean, n.rstd) = at::native_layer_norm(n.sum, {d}, lw, lb, eps);
    return n;
  }
  n.mean = at::empty({2, T}, x.options().dtype(at::kFloat));
  float* mean = n.mean.data_ptr<float>();
  n.h = at::empty({T, d}, x.options());
  if (pending) {
    n.sum = at::empty({T, d}, x.options());
    check(mcclAddLayerNormForward(x.data_ptr(), pending->data_ptr(), lw.data_ptr(), lb.data_ptr(), n.sum.data_ptr(), n.h.data_ptr(), mean,
                                  mean + T, T, (int)d, (float)eps, streamOf(x)), "mcclAddLayerNormForward");
  } else {
    n.sum = at::alias(x);
    check(mcclLayerNormForward(x.data_ptr(), lw.data_ptr(), lb.data_ptr(), n.h.data_ptr(), mean, mean + T, T, (int)d, (float)eps, streamOf(x)),
          "mcclLayerNormForward");
  }
  counters().norm++;
  return n;
}

// out = [+] column sums of up to three [T, d] matrices, a gradient each.
void columnSums(GradSink& sink, std::initializer_list<Tensor> x, const VectorGrads& out) {
  const Tensor& first = *x.begin();
  const int64_t T = first.size(0), d = first.size(1);
  const void* in[3];
  void* to[3];
  int n = 0;
  for (const Tensor& t : x) { in[n] = t.data_ptr(); to[n] = out.t[n].data_ptr(); ++n; }
  Tensor scratch = columnScratch(first, T, d, n);
  check(mcclColumnSums(in, to, n, out.direct, scratch.data_ptr<float>(), T, (int)d, d, streamOf(first)), "mcclColumnSums");
}

// Gradient of a norm's sum from those of its result (the sum of `parts`, added up in their order with a rounding each) and, where
// defined, of the residual stream; *dw, *db and, with `bias`, *dbias (column sums of the whole) as they are to be returned.
Tensor normBackward(GradSink& sink, const Tensor& sum, std::initializer_list<Tensor> parts, const Tensor& dres, const Tensor& lw, const Tensor& lb,
                    const Tensor& mean, const Tensor& rstd, const Tensor& bias, Tensor* dw, Tensor* db, Tensor* dbias) {
  const int64_t T = sum.size(0), d = sum.size(1);
  const bool own = !rstd.defined();
  Tensor partial = at::empty({(int64_t)mcclLayerNormPartials(T) * 3 * d}, mean.options()), dx, dn;
  const float *m = mean.data_ptr<float>(), *r = own ? m + T : rstd.data_ptr<float>();
  const void* dh[3] = {};
  int n = 0;
  for (const Tensor& p : parts) dh[n++] = p.data_ptr();
  if (own) {
    dx = at::empty({T, d}, sum.options());
  } else {
    Tensor dy = *parts.begin();
    for (const Tensor& p : parts) if (!p.is_same(dy)) dy.add_(p);
    dn = std::get<0>(at::native_layer_norm_backward(dy, sum, {d}, mean, rstd, lw, lb, {true, false, false}));
    dx = dres.defined() ? at::empty({T, d}, sum.options()) : dn;
  }
  void* res = dres.defined() ? dres.data_ptr() : nullptr;
  auto run = [&](const VectorGrads& g, void* dcol) {
    if (own) {
      check(mcclAddLayerNormBackward(sum.data_ptr(), dh[0], dh[1], dh[2], res, lw.data_ptr(), m, r, dx.data_ptr(), g.t[0].data_ptr(),
                                     g.t[1].data_ptr(), dcol, g.direct, partial.data_ptr<float>(), T, (int)d, streamOf(sum)),
            "mcclAddLayerNormBackward");
    } else {
      check(mcclLayerNormBackwardTail(sum.data_ptr(), dh[0], dn.data_ptr(), res, m, r, dx.data_ptr(), g.t[0].data_ptr(), g.t[1].data_ptr(), dcol,
                                      g.direct, partial.data_ptr<float>(), T, (int)d, streamOf(sum)), "mcclLayerNormBackwardTail");
    }
    *dw = g.ret(0);
    *db = g.ret(1);
  };
  if (bias.defined() && dres.defined()) {
    VectorGrads g(sink, {&lw, &lb, &bias});
    run(g, g.t[2].data_ptr());
    *dbias = g.ret(2);
  } else {
    VectorGrads g(sink, {&lw, &lb});
    run(g, nullptr);
    if (bias.defined()) {
      VectorGrads b(sink, {&bias});
      columnSums(sink, {dx}, b);
      *dbias = b.ret(0);
    }
  }
  counters().norm += 2;
  return dx;
}

// ---- first half: (residual, pending) -> residual sum, norm, q, k, v -----------------------------------------------------
struct BlockInFn : torch::autograd::Function<BlockInFn> {
  // Outputs: residual [T, d], q, k, v [b, h, s, hd].
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& pending, const OptTensor& pendingBias, const Tensor& lw,
                               const Tensor& lb, const Tensor& wq, const Tensor& bq, const Tensor& wk, const Tensor& bk, const Tensor& wv,
                               const Tensor& bv, int64_t b, int64_t s, int64_t heads, double eps, bool sink) {
    Below below;
    const int64_t d = x.size(1), hd = d / heads;
    const Norm n = addNorm(x, pending ? &*pending : nullptr, lw, lb, eps);
    const Tensor& h = n.h;
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
    ctx->save_for_backward({pending ? n.sum : x, h, n.mean, n.rstd, lw, lb, wq, bq, wk, bk, wv, bv, pendingBias ? *pendingBias : Tensor()});
    ctx->saved_data["sink"] = sink;
    ctx->saved_data["pending"] = pending.has_value();
    return {n.sum, q, k, v};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &sum = saved[0], &h = saved[1], &mean = saved[2], &rstd = saved[3], &lw = saved[4], &lb = saved[5], &wq = saved[6],
                 &bq = saved[7], &wk = saved[8], &bk = saved[9], &wv = saved[10], &bv = saved[11], &pb = saved[12];
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = h.size(0), d = h.size(1);
    const Tensor dq = fromHeads(g[1], T, d), dk = fromHeads(g[2], T, d), dv = fromHeads(g[3], T, d);
    variable_list ret(17);
    VectorGrads db(sink, {&bv, &bk, &bq});
    // Weight gradients: where their buffers lie next to each other the three gradients are laid side by side on the pass that sums
    // their columns, and one product fills all of them (the same sums: a product's columns do not meet).
    const Tensor gv = sink.buffer(wv), gk = sink.buffer(wk), gq = sink.buffer(wq);
    Tensor g3 = gv.defined() && gk.defined() && gq.defined() ? adjacent(gv, gk, gq) : Tensor();
    if (g3.defined()) {
      Tensor d3 = at::empty({T, 3 * d}, h.options()), scratch = columnScratch(h, T, d, 3);
      const void* in[3] = {dv.data_ptr(), dk.data_ptr(), dq.data_ptr()};
      void* out[3] = {db.t[0].data_ptr(), db.t[1].data_ptr(), db.t[2].data_ptr()};
      check(mcclPackColumnSums(in, d3.data_ptr(), out, 3, db.direct, scratch.data_ptr<float>(), T, (int)d, streamOf(h)), "mcclPackColumnSums");
      at::addmm_out(g3, g3, d3.t(), h);
    } else {
      columnSums(sink, {dv, dk, dq}, db);
      weightGrad(sink, wv, dv, h, &ret[9]);
      weightGrad(sink, wk, dk, h, &ret[7]);
      weightGrad(sink, wq, dq, h, &ret[5]);
    }
    ret[6] = db.ret(2); ret[8] = db.ret(1); ret[10] = db.ret(0);
    // The norm's gradient stays three products, each rounded: as one product of three times the depth it is faster (34 us for
    // 3 x 15 at 8192 x 1024) but rounds once, and every number behind it differs from the separate operations'.
    ret[0] = normBackward(sink, sum, {at::mm(dv, wv), at::mm(dk, wk), at::mm(dq, wq)}, rows2d(g[0], T, d), lw, lb, mean, rstd, pb, &ret[3], &ret[4],
                          &ret[2]);
    if (ctx->saved_data["pending"].toBool()) ret[1] = ret[0];
    return once(std::move(ret));
  }
};

// ---- second half: attention output and residual -> residual sum, MLP output ---------------------------------------------
struct BlockOutFn : torch::autograd::Function<BlockOutFn> {
  // Outputs: residual after attention [T, d], MLP output (with its bias) [T, d].  outBiasHere: the bias gradient of the down
  // projection is taken by this node and not by the one that adds its output.
  static variable_list forward(AutogradContext* ctx, const Tensor& a, const Tensor& res, const Tensor& wo, const Tensor& bo, const Tensor& lw,
                               const Tensor& lb, const Tensor& wf, const Tensor& bf, const Tensor& wd, const Tensor& bd, bool outBiasHere,
                               double eps, bool sink) {
    Below below;
    const int64_t T = res.size(0), d = res.size(1);
    mcclStream_t s = streamOf(res);
    Tensor a2 = fromHeads(a, T, d);
    Tensor p = at::linear(a2, wo, bo);
    const Norm n = addNorm(res, &p, lw, lb, eps);
    Tensor u = at::linear(n.h, wf, bf);
    Tensor act = at::empty(u.sizes(), u.options());
    check(mcclGeluForward(u.data_ptr(), act.data_ptr(), u.numel(), s), "mcclGeluForward");
    Tensor y = at::linear(act, wd, bd);
    ctx->save_for_backward({a2, n.sum, n.h, n.mean, n.rstd, u, act, wo, bo, lw, lb, wf, bf, wd, bd});
    ctx->saved_data["sink"] = sink;
    ctx->saved_data["bias"] = outBiasHere;
    ctx->saved_data["b"] = a.size(0);
    ctx->saved_data["h"] = a.size(1);
    return {n.sum, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &a2 = saved[0], &x1 = saved[1], &h = saved[2], &mean = saved[3], &rstd = saved[4], &u = saved[5], &act = saved[6], &wo = saved[7],
                 &bo = saved[8], &lw = saved[9], &lb = saved[10], &wf = saved[11], &bf = saved[12], &wd = saved[13], &bd = saved[14];
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    const int64_t T = h.size(0), d = h.size(1), f = u.size(1), b = ctx->saved_data["b"].toInt(), heads = ctx->saved_data["h"].toInt();
    variable_list ret(14);
    const Tensor dy = rows2d(g[1], T, d), dres = rows2d(g[0], T, d);
    if (ctx->saved_data["bias"].toBool()) {
      VectorGrads db(sink, {&bd});
      columnSums(sink, {dy}, db);
      ret[9] = db.ret(0);
    }
    Tensor du = at::mm(dy, wd);
    weightGrad(sink, wd, dy, act, &ret[8]);
    {
      VectorGrads db(sink, {&bf});
      Tensor scratch = columnScratch(h, T, f, 1);
      check(mcclGeluBackward(u.data_ptr(), du.data_ptr(), du.data_ptr(), db.t[0].data_ptr(), db.direct, scratch.data_ptr<float>(), T, (int)f,
                             streamOf(h)), "mcclGeluBackward");
      ret[7] = db.ret(0);
    }
    Tensor dh = at::mm(du, wf);
    weightGrad(sink, wf, du, h, &ret[6]);
    const Tensor dx = normBackward(sink, x1, {dh}, dres, lw, lb, mean, rstd, bo, &ret[4], &ret[5], &ret[3]);
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
                        const Tensor& lb, double eps, bool sink) {
    Below below;
    const Norm n = addNorm(x, &pending, lw, lb, eps);
    ctx->save_for_backward({n.sum, n.mean, n.rstd, lw, lb, pendingBias ? *pendingBias : Tensor()});
    ctx->saved_data["sink"] = sink;
    return n.h;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto saved = ctx->get_saved_variables();
    const Tensor &sum = saved[0];
    Below below;
    c10::cuda::CUDAGuard guard(sum.device());
    GradSink sink(ctx->saved_data["sink"].toBool());
    variable_list ret(8);
    ret[0] = normBackward(sink, sum, {rows2d(g[0], sum.size(0), sum.size(1))}, Tensor(), saved[3], saved[4], saved[1], saved[2], saved[5], &ret[3], &ret[4],
                          &ret[2]);
    ret[1] = ret[0];
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
        // Too many tokens for the kernel's scan: the sorting form of the tensor library, which does not look whether an index is
        // in the table; those that are not (their rows were NaN) go to a row behind it.
        Tensor i = idx.view({T});
        i = at::where(at::logical_and(i.ge(0), i.lt(V)), i, V);
        ret[1] = at::embedding_dense_backward(dy, i, V + 1, -1, false).narrow(0, 0, V);
        if (withPos) {
          ret[2] = at::zeros(pos.sizes(), pos.options());
          ret[2].narrow(0, 0, seq).copy_(dy.view({T / seq, seq, d}).sum(0));
        }
        return once(std::move(ret));
      }
    }
    Tensor work = at::empty({mcclEmbeddingWork(T, V, (int)d)}, dy.options().dtype(at::kByte));
    check(mcclEmbeddingBackwardWork(idx.data_ptr<int64_t>(), dy.data_ptr(), dt.data_ptr(), withPos ? dp.data_ptr() : nullptr, work.data_ptr(), T,
                                    (int)seq, V, (int)d, streamOf(dy)), "mcclEmbeddingBackwardWork");
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
    Below below;
    c10::cuda::CUDAGuard guard(h.device());
    // Their gradient is written over the logits; a second pass over a retained graph works them out again.
    Tensor logits = ctx->saved_data.count("spent") ? at::linear(h, w) : saved[3];
    ctx->saved_data["spent"] = true;
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
  if (pendingBias && (!pending || !plainBf16(*pendingBias, x) || !shaped(*pendingBias, {d}))) return py::none();
  for (int i : {0, 1, 3, 5, 7, 9, 10, 11, 15}) if (!shaped(p[i], {d})) return py::none();
  for (int i : {2, 4, 6, 8}) if (!shaped(p[i], {d, d})) return py::none();
  if (!shaped(p[12], {f, d}) || !shaped(p[13], {f}) || !shaped(p[14], {d, f})) return py::none();
  c10::cuda::CUDAGuard guard(x.device());
  variable_list in = BlockInFn::apply(x, pending, pendingBias, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], b, s, heads, eps, sink);
  Tensor a = at::scaled_dot_product_attention(in[1], in[2], in[3], {}, 0.0, true);
  variable_list out = BlockOutFn::apply(a, in[0], p[8], p[9], p[10], p[11], p[12], p[13], p[14], p[15], outBiasHere, eps, sink);
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
  return py::cast(FinalNormFn::apply(x, pending, pendingBias, w, b, eps, sink));
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
