/*
 * mccl-b200 compute entry points that go with the collectives: the tcgen05 GEMM and its fused tensor-parallel
 * forms, the fused expert-parallel token exchange, and the kernels of the data-parallel training step (fused
 * AdamW with global-norm clipping, sum of squares, cross-entropy, LayerNorm).  sm_100a only; every pointer is a
 * device pointer on the current device unless stated otherwise; calls are enqueued on `stream`.
 * None of these has a counterpart in the reference (a communication library without compute or model code).
 */
#ifndef MCCL_OPS_H_
#define MCCL_OPS_H_

#include "mccl.h"

#ifdef __cplusplus
extern "C" {
#endif

/* ---- bf16 GEMM on the 5th-generation tensor cores: C[M,N] = act(A[M,K] * B[N,K]^T) --------------------------- */
#define MCCL_EPILOGUE_NONE 0
#define MCCL_EPILOGUE_SILU 1
/* M % 128 == 0, N % 64 == 0, K % 64 == 0.  maxCtas = 0: one CTA per SM. */
mcclResult_t mcclTpGemm(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, int maxCtas, mcclStream_t stream);
/* The same product by pairs of SMs on 256-row tiles (M % 256 == 0). */
mcclResult_t mcclTpGemm2(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, int maxCtas, mcclStream_t stream);
/* The same by the form the shape allows; pre (nullable, [M, N]): the sums before the activation. */
mcclResult_t mcclTpGemmKeepPre(const void* A, const void* B, void* C, void* pre, int M, int N, int K, int epilogue, mcclStream_t stream);
/* Error code the last GEMM kernel on the current device recorded (0 = none); reading clears it. */
int mcclTpGemmLastError(void);

/* Fused all-gather -> GEMM -> activation.  xShard [M/n, K] in symmetric memory, xFull [M, K] local workspace,
 * W [N, K] local weight shard, out [M, N], flags >= 16 uint64 of device memory.  Collective over comm. */
mcclResult_t mcclTpAllGatherGemm(mcclComm_t comm, const void* xShard, void* xFull, const void* W, void* out, void* flags,
                                 int M, int N, int K, int epilogue, mcclStream_t stream);
/* Fused GEMM -> reduce-scatter over rows.  H [M, K], W [N, K], partial [M, N] and flags (16 + M/128 + M/128 uint64,
 * zeroed once) in symmetric memory, out [M/n, N], accum [M/n, N] fp32; callIndex = 1, 2, ... per flags buffer. */
mcclResult_t mcclTpGemmReduceScatter(mcclComm_t comm, const void* H, const void* W, void* partial, void* flags, void* out,
                                     float* accum, int M, int N, int K, uint64_t callIndex, mcclStream_t stream);

/* ---- expert-parallel token exchange fused with the routing gather / scatter --------------------------------------- */
/* exchange: symmetric memory, [ranks][expertsPerRank][capacity][rowBytes] on every rank.  flat[t] = expert * capacity +
 * slot of token t, negative for a dropped token.  scale (nullable): one float per token. */
mcclResult_t mcclMoeScatter(mcclComm_t comm, const void* tokens, const int32_t* flat, const float* scale, void* exchange,
                            int nTokens, int rowBytes, int expertsPerRank, int capacity, mcclDataType_t dt, mcclStream_t stream);
mcclResult_t mcclMoeGather(mcclComm_t comm, const void* exchange, const int32_t* flat, const float* scale, void* out,
                           int nTokens, int rowBytes, int expertsPerRank, int capacity, mcclDataType_t dt, mcclStream_t stream);

/* ---- routing and token movement with all experts on this GPU (bf16 rows of d elements, d % 8 == 0) ------------------- */
/* Top-1 routing from logits [tokens, experts]: gate (fp32, rounded to bf16), log-sum-exp, flat[t] = expert * capacity + slot in
 * token order or -1; inverse[expert * capacity + slot] = t and kept[expert] (both nullable).  At most mcclMoeRouteMaxExperts()
 * experts; scratch: mcclMoeRouteScratch() ints. */
int          mcclMoeRouteMaxExperts(void);
int64_t      mcclMoeRouteScratch(int tokens, int experts);
mcclResult_t mcclMoeRoute(const void* logits, int tokens, int experts, int capacity, float* gate, float* lse, int32_t* flat,
                          int32_t* inverse, int32_t* kept, int32_t* scratch, mcclStream_t stream);
/* slots[s] = rows[inverse[s]], zero where empty. */
mcclResult_t mcclMoeFillSlots(const void* rows, const int32_t* inverse, const int32_t* kept, void* slots, int experts, int capacity,
                              int d, mcclStream_t stream);
/* out[t] = gate[t] * slots[flat[t]], zero for a dropped token. */
mcclResult_t mcclMoeCombine(const void* slots, const int32_t* flat, const float* gate, void* out, int tokens, int d, mcclStream_t stream);
mcclResult_t mcclMoeCombineBackward(const void* dy, const void* slots, const int32_t* inverse, const int32_t* kept, const float* gate,
                                    void* dslots, float* dgate, int experts, int capacity, int d, mcclStream_t stream);
/* dlogits through the softmax of the gate and dx = dslots[flat] + dlogits router (router null: without the second term; d = 0:
 * dlogits only). */
mcclResult_t mcclMoeTokenBackward(const void* dslots, const int32_t* flat, const float* dgate, const void* logits, const float* lse,
                                  const void* router, void* dlogits, void* dx, int tokens, int experts, int capacity, int d,
                                  mcclStream_t stream);

/* ---- activations over n bf16 values (16-byte aligned) ---------------------------------------------------------------- */
mcclResult_t mcclSiluForward(const void* x, void* y, int64_t n, mcclStream_t stream);
mcclResult_t mcclSiluBackward(const void* x, const void* dy, void* dx, int64_t n, mcclStream_t stream);
mcclResult_t mcclSiluForwardBackward(const void* x, const void* dy, void* y, void* dx, int64_t n, mcclStream_t stream);
mcclResult_t mcclSwigluForward(const void* gate, const void* up, void* y, int64_t n, mcclStream_t stream);
mcclResult_t mcclSwigluBackward(const void* gate, const void* up, const void* dy, void* y, void* dgate, void* dup, int64_t n,
                                mcclStream_t stream);
mcclResult_t mcclGeluForward(const void* x, void* y, int64_t n, mcclStream_t stream);
/* dx = dy * gelu'(x) over [rows, D] and dbias (nullable) = [+] its column sums; scratch: mcclColumnSumScratch(rows, D, 1) floats. */
mcclResult_t mcclGeluBackward(const void* x, const void* dy, void* dx, void* dbias, int accumulate, float* scratch, int64_t rows, int D,
                              mcclStream_t stream);
/* out[i] = [+] column sums of x[i], n <= 3 matrices [rows, D] with rows ld elements apart. */
int64_t      mcclColumnSumScratch(int64_t rows, int D, int segments);
mcclResult_t mcclColumnSums(const void* const* x, void* const* out, int n, int accumulate, float* scratch, int64_t rows, int D, int64_t ld,
                            mcclStream_t stream);

/* ---- embedding: out[t] = table[idx[t]] + pos[t % seq] (pos nullable); the backward pass adds into the gradients ---------- */
mcclResult_t mcclEmbeddingForward(const int64_t* idx, const void* table, const void* pos, void* out, int64_t tokens, int seq, int64_t vocab,
                                  int D, mcclStream_t stream);
/* tokens <= mcclEmbeddingMaxTokens(), D <= 4096; work: mcclEmbeddingWork() bytes, 16-byte aligned. */
int          mcclEmbeddingMaxTokens(void);
int64_t      mcclEmbeddingWork(int64_t tokens, int64_t vocab, int D);
mcclResult_t mcclEmbeddingBackwardWork(const int64_t* idx, const void* dy, void* tableGrad, void* posGrad, void* work, int64_t tokens, int seq,
                                       int64_t vocab, int D, mcclStream_t stream);
/* The same with work memory of its own, in the stream's order (count: vocab ints, not used). */
mcclResult_t mcclEmbeddingBackward(const int64_t* idx, const void* dy, void* tableGrad, void* posGrad, int32_t* count, int64_t tokens, int seq,
                                   int64_t vocab, int D, mcclStream_t stream);

/* ---- rotary position embedding: pairs (i, i + hd/2) of every head turned by position x theta^(-i / (hd/2)) ---------------- */
/* src: [batch, seq, heads, hd] at element strides sb, ss, sh (last one 1); dst: contiguous [batch, seq, heads, hd], may be src where
 * that is contiguous too; inverse: turn back (the backward pass).  Two arrays in one launch (the second may be null). */
mcclResult_t mcclRope(const void* src0, const void* src1, void* dst0, void* dst1, int batch, int seq, int heads, int hd, int64_t sb,
                      int64_t ss, int64_t sh, float theta, int inverse, mcclStream_t stream);

/* ---- training-step kernels (bf16 parameters and gradients, fp32 state) --------------------------------------------- */
/* AdamW on n elements; normSq / maxNorm (nullable / 0): clip by the global gradient norm held on the device. */
mcclResult_t mcclFusedAdamW(void* param, float* master, float* expAvg, float* expAvgSq, const void* grad, uint64_t n, float lr,
                            float beta1, float beta2, float eps, float weightDecay, float gradScale, int step, int zeroGrad,
                            const float* normSq, float maxNorm, mcclStream_t stream);
/* The same step with {lr, 1 - beta1^t, sqrt(1 - beta2^t)} read from the device array `hyper` when the kernel runs, so a
   launch recorded in a CUDA graph follows the schedule on every replay. */
mcclResult_t mcclFusedAdamWDeviceHyper(void* param, float* master, float* expAvg, float* expAvgSq, const void* grad, uint64_t n,
                                       const float* hyper, float beta1, float beta2, float eps, float weightDecay, float gradScale,
                                       int zeroGrad, const float* normSq, float maxNorm, mcclStream_t stream);
uint64_t     mcclSumSquaresScratchFloats(uint64_t n);
/* out = [out +] sum(x^2) over n bf16 values; scratch: mcclSumSquaresScratchFloats(n) floats, first word zero. */
mcclResult_t mcclSumSquaresBf16(const void* x, uint64_t n, float* scratch, uint64_t scratchFloats, float* out, int accumulate,
                                mcclStream_t stream);
/* Cross-entropy over bf16 logits [rows, ld] (vocab <= ld): per-row loss and log-sum-exp; backward in place. */
mcclResult_t mcclCrossEntropyForward(const void* logits, int64_t rows, int64_t ld, int vocab, const int64_t* targets, float* loss,
                                     float* lse, mcclStream_t stream);
/* The same with the mean of the rows' losses in *mean: over all rows, or, with inverse (nullable), over those whose target is a
 * column; one over their number goes to *inverse, which the backward pass takes. */
mcclResult_t mcclCrossEntropyMean(const void* logits, int64_t rows, int64_t ld, int vocab, const int64_t* targets, float* loss, float* lse,
                                  float* mean, float* inverse, mcclStream_t stream);
mcclResult_t mcclCrossEntropyMeanBackward(void* logits, int64_t rows, int64_t ld, int vocab, int width, const int64_t* targets,
                                          const float* lse, const float* gradOut, const float* inverse, mcclStream_t stream);
mcclResult_t mcclCrossEntropyBackward(void* logits, int64_t rows, int64_t ld, int vocab, int width, const int64_t* targets,
                                      const float* lse, const float* gradOut, mcclStream_t stream);
/* LayerNorm over bf16 rows of D elements, D % 8 == 0 and D <= 4096.  The backward passes need partial:
 * mcclLayerNormPartials(rows) x 2 x D (3 x D for the Add form) floats of work memory. */
int          mcclLayerNormPartials(int64_t rows);
mcclResult_t mcclLayerNormForward(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int64_t rows,
                                  int D, float eps, mcclStream_t stream);
mcclResult_t mcclLayerNormBackward(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd, void* dx,
                                   void* dgamma, void* dbeta, float* partial, int64_t rows, int D, mcclStream_t stream);
/* With the residual add of a pre-norm block: sum = x + delta, y = LayerNorm(sum).  Backward (x: the sum): dx = d sum of the norm +
 * dres; dcol (nullable, needs dres) = column sums of dx; accumulate: dgamma, dbeta and dcol are added to what is there. */
mcclResult_t mcclAddLayerNormForward(const void* x, const void* delta, const void* gamma, const void* beta, void* sum, void* y, float* mean,
                                     float* rstd, int64_t rows, int D, float eps, mcclStream_t stream);
mcclResult_t mcclPackColumnSums(const void* const* x, void* packed, void* const* out, int n, int accumulate, float* scratch, int64_t rows,
                                int D, mcclStream_t stream);
mcclResult_t mcclAddLayerNormBackward(const void* x, const void* dy, const void* dy2, const void* dy3, const void* dres, const void* gamma,
                                      const float* mean, const float* rstd, void* dx, void* dgamma, void* dbeta, void* dcol, int accumulate, float* partial,
                                      int64_t rows, int D, mcclStream_t stream);
/* What is left of the backward pass when dn, the gradient through the norm, is there: dx = dn + dres (both nullable: dx is dn),
 * dgamma, dbeta and dcol (nullable).  partial as in the Add form. */
mcclResult_t mcclLayerNormBackwardTail(const void* x, const void* dy, const void* dn, const void* dres, const float* mean, const float* rstd,
                                       void* dx, void* dgamma, void* dbeta, void* dcol, int accumulate, float* partial, int64_t rows, int D,
                                       mcclStream_t stream);
/* RMSNorm, y = bf16(x * rstd) * gamma; delta and sum (nullable) as above; dres nullable. */
mcclResult_t mcclRmsNormForward(const void* x, const void* delta, const void* gamma, void* sum, void* y, float* rstd, int64_t rows, int D,
                                float eps, mcclStream_t stream);
mcclResult_t mcclRmsNormBackward(const void* x, const void* dy, const void* dy2, const void* dy3, const void* dres, const void* gamma,
                                 const float* rstd, void* dx, void* dgamma, int accumulate, float* partial, int64_t rows, int D, mcclStream_t stream);

#ifdef __cplusplus
}
#endif
#endif /* MCCL_OPS_H_ */
