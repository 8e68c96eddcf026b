// Helpers of the decoders' nodes.
#pragma once

#include "gradsink.h"

namespace mccl_torch {

using OptTensor = std::optional<Tensor>;

inline Tensor columnScratch(const Tensor& like, int64_t rows, int64_t d, int n) {
  return at::empty({mcclColumnSumScratch(rows, (int)d, n)}, like.options().dtype(at::kFloat));
}

inline Tensor rows2d(const Tensor& g, int64_t T, int64_t d) {
  Tensor r = g.reshape({T, d});
  return r.is_contiguous() && aligned16(r) ? r : r.clone(at::MemoryFormat::Contiguous);
}

// [b, h, s, hd] (any layout) -> [b s, h hd]; no copy when the memory is laid out that way.
inline Tensor fromHeads(const Tensor& a, int64_t T, int64_t d) { return rows2d(a.transpose(1, 2), T, d); }

inline bool plainBf16(const Tensor& t, const Tensor& like) {
  return ordinary(t) && t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.device() == like.device() && t.is_contiguous() && aligned16(t);
}

inline bool usable(const Tensor& x, const std::vector<Tensor>& params) {
  if (recorded() || !plainBf16(x, x) || x.size(-1) % 8 || x.size(-1) > 4096 || x.numel() == 0) return false;
  for (const Tensor& p : params) if (!plainBf16(p, x)) return false;
  return true;
}

inline bool shaped(const Tensor& t, at::IntArrayRef sizes) { return t.sizes() == sizes; }

// With attention by matrix products alone (the other kinds switched off) a model can be differentiated twice: the nodes,
// which cannot, leave it to the tensor operations.
inline bool attentionOnce() {
  auto& c = at::globalContext();
  return c.userEnabledFlashSDP() || c.userEnabledMemEfficientSDP() || c.userEnabledCuDNNSDP();
}

}  // namespace mccl_torch
