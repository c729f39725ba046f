/* Element-wise parts of a decoder block on one GPU: bf16 in and out, fp32 arithmetic. Matrices are row-major and contiguous,
 * pointers 16-byte aligned. The Python models call these between the fused matmul + collective operators. */
#ifndef HCCL_NN_H_
#define HCCL_NN_H_

#include <cuda_runtime.h>
#include <stdint.h>
#include "hccl_types.h"

#ifdef __cplusplus
extern "C" {
#endif

/* y[rows, hidden] = x * rsqrt(mean(x^2) + eps) * w; rstd[rows] receives the reciprocal norms for the backward pass.
 * hidden: a multiple of 8, at most 12288. */
HcclResult HcclRmsNorm(const void *x, const void *w, void *y, float *rstd, uint64_t rows, uint64_t hidden, float eps, cudaStream_t stream);
/* The same, and copies of x and w: what the backward pass reads where x or w may be changed in between. */
HcclResult HcclRmsNormKeep(const void *x, const void *w, void *y, float *rstd, void *xKept, void *wKept, uint64_t rows, uint64_t hidden, float eps, cudaStream_t stream);
/* sum = x + d, and the norm of that sum; wKept may be null. */
HcclResult HcclRmsNormAdd(const void *x, const void *d, const void *w, void *sum, void *y, float *rstd, void *wKept, uint64_t rows, uint64_t hidden, float eps, cudaStream_t stream);
/* Rows of the fp32 workspace `partial` [parts, hidden] that HcclRmsNormBwd needs. Up to 1024 columns it may also be aligned to 4 bytes alone. */
uint64_t HcclRmsNormBwdParts(uint64_t rows, uint64_t hidden);
HcclResult HcclRmsNormBwd(const void *dy, const void *x, const void *w, const float *rstd, void *dx, void *dw, float *partial, uint64_t rows, uint64_t hidden,
                          cudaStream_t stream);
/* The same with dSum[rows, hidden] added to dx: the gradient that reached x (the sum) past the norm. Null: nothing is added. */
HcclResult HcclRmsNormBwdAdd(const void *dy, const void *x, const void *w, const float *rstd, const void *dSum, void *dx, void *dw, float *partial, uint64_t rows,
                             uint64_t hidden, cudaStream_t stream);
/* qkv[tokens, (qHeads + 2 kvHeads) * headDim] -> q, k rotated (pairs are element j and j + headDim / 2) and v, each
 * [tokens, heads, headDim]; cos / sin: fp32 [seq, headDim / 2], token t takes row t % seq. headDim: a multiple of 16.
 * backward != 0: gradients of q, k, v -> gradient of qkv. */
HcclResult HcclRopeQkv(void *qkv, void *q, void *k, void *v, const float *cosT, const float *sinT, uint64_t tokens, uint64_t seq, uint32_t qHeads, uint32_t kvHeads,
                       uint32_t headDim, int backward, cudaStream_t stream);
/* Gradient of causal attention by the packed projection qkv[batch * seq, (qHeads + 2 kvHeads) * headDim], whose q and k HcclRopeQkv rotates: dQkv from dO and o[batch * seq, qHeads * headDim]
 * and lse[batch, qHeads, seq], the logarithms of the sums of exp(q k / sqrt(headDim)). Query head h reads key head h / (qHeads / kvHeads). headDim: 32 or 64.
 * HcclAttentionBwdSuits: whether this kernel, made for short sequences, is the better choice. */
int HcclAttentionBwdSuits(uint64_t batch, uint64_t seq, uint32_t qHeads, uint32_t kvHeads, uint32_t headDim);
HcclResult HcclAttentionBwd(const void *dO, const void *qkv, const void *o, const float *lse, void *dQkv, const float *cosT, const float *sinT, uint64_t batch, uint64_t seq,
                            uint32_t qHeads, uint32_t kvHeads, uint32_t headDim, cudaStream_t stream);
/* h[rows, ffn] = silu(gate) * up with gateUp[rows, 2 ffn] = [gate | up]. ffn: a multiple of 8. */
HcclResult HcclSwiGlu(const void *gateUp, void *h, uint64_t rows, uint64_t ffn, cudaStream_t stream);
HcclResult HcclSwiGluBwd(const void *dh, const void *gateUp, void *dGateUp, uint64_t rows, uint64_t ffn, cudaStream_t stream);
/* Cross entropy over a vocabulary shard. step 0: rowMax[rows]. step 1: packed[0][rows] = sum exp(logit - rowMax), packed[1][rows] =
 * target logit - rowMax, 0 where the target lies outside [vocabStart, vocabStart + vocab). step 2: grad = (exp(logit - rowMax) /
 * packed[0] - onehot(target)) * gradOut[0] / rows. The maxima and sums over the shards are the caller's, between the steps. */
HcclResult HcclXent(int step, const void *logits, const int64_t *targets, int64_t vocabStart, float *rowMax, float *packed, const float *gradOut, void *grad, uint64_t rows,
                    uint64_t vocab, cudaStream_t stream);

/* The same on one rank, up to the loss: rowMax and packed as steps 0 and 1 leave them, rowLoss[rows] = log(packed[0]) - packed[1], loss = their mean; keptLogits and keptTargets
 * (either may be null) receive copies. */
HcclResult HcclXentLoss(const void *logits, const int64_t *targets, int64_t vocabStart, float *rowMax, float *packed, float *rowLoss, void *keptLogits, int64_t *keptTargets, float *loss,
                        uint64_t rows, uint64_t vocab, cudaStream_t stream);
/* grad[vocab, hidden] = sums of the rows of dy[tokens, hidden] by their ids (negative ones count from the end; others outside are left out), zeros elsewhere. tokens: at most
 * HcclEmbeddingGradTokens(); hidden: a multiple of 8. */
uint64_t HcclEmbeddingGradTokens(void);
HcclResult HcclEmbeddingGrad(const int64_t *ids, const void *dy, void *grad, uint64_t tokens, uint64_t hidden, uint64_t vocab, cudaStream_t stream);

#ifdef __cplusplus
}
#endif
#endif
