/*
 * ttcb200_mlp.h -- device kernels of the learned schedule selector (a 3-layer fp32 MLP that ranks
 * transposition schedules). No counterpart in TTC, which times every generated variant instead
 * (ttc.py:847-1022). All matrices are row-major fp32 device arrays; every call is stream-ordered and
 * returns a ttcb_status.
 */
#ifndef TTCB200_MLP_H
#define TTCB200_MLP_H

#include "ttcb200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* C[M x N] = op(A) * op(B) (+ bias[N]) (then ReLU if relu != 0), op = transpose when trans* != 0.
 * op(A) is M x K, op(B) is K x N; lda/ldb/ldc are row strides of the stored matrices. */
ttcb_status ttcb_mlp_gemm(int transA, int transB, int M, int N, int K, const float* A, int lda, const float* B,
                          int ldb, float* C, int ldc, const float* bias, int relu, ttcb_stream_t stream);

/* dZ = dY * (Y > 0), elementwise over n values (backward of ReLU, given the ReLU output Y). */
ttcb_status ttcb_mlp_relu_grad(const float* Y, const float* dY, float* dZ, int n, ttcb_stream_t stream);

/* out[N] = sum over rows of X[M x N] (the bias gradient). */
ttcb_status ttcb_mlp_colsum(const float* X, int M, int N, float* out, ttcb_stream_t stream);

/* Mean squared error: dpred = 2 (pred - target) / n, loss[0] = mean (pred - target)^2. */
ttcb_status ttcb_mlp_mse(const float* pred, const float* target, int n, float* dpred, float* loss,
                         ttcb_stream_t stream);

/* One Adam step (Kingma & Ba, 2015) on n parameters, step t >= 1. */
ttcb_status ttcb_mlp_adam(float* param, const float* grad, float* m, float* v, int n, float lr, float beta1,
                          float beta2, float eps, int t, ttcb_stream_t stream);

/* The same step with L2 weight decay: the gradient used is grad + weight_decay * param. */
ttcb_status ttcb_mlp_adam_l2(float* param, const float* grad, float* m, float* v, int n, float lr, float beta1,
                             float beta2, float eps, float weight_decay, int t, ttcb_stream_t stream);

/* The same step on `count` parameter tensors (host arrays of device pointers and sizes) in one launch. */
ttcb_status ttcb_mlp_adam_multi(int count, float* const* param, const float* const* grad, float* const* m,
                                float* const* v, const int* n, float lr, float beta1, float beta2, float eps,
                                float weight_decay, int t, ttcb_stream_t stream);

/* The whole network (nin -> 128 -> 128 -> 1, ReLU between the layers) in one launch. params: host array of the
 * six device tensors W1 [nin x 128], b1, W2 [128 x 128], b2, W3 [128], b3 [1]. X is rows x nin; H1 and H2
 * [rows x 128] receive the hidden layers' outputs, out [rows] the network's. At most
 * ttcb_mlp_passes_max_features() features. */
ttcb_status ttcb_mlp_forward(int rows, int nin, const float* X, const float* const* params, float* H1, float* H2,
                             float* out, ttcb_stream_t stream);

/* Its gradients, given dout [rows] = d loss / d out: grads holds W1, b1, W2, b2, W3 and b3's one after the other.
 * workspace: ttcb_mlp_backward_workspace(rows, nin) bytes of device memory, free again after the call (in
 * stream order). */
ttcb_status ttcb_mlp_backward(int rows, int nin, const float* X, const float* const* params, const float* H1,
                              const float* H2, const float* dout, float* grads, void* workspace, ttcb_stream_t stream);
size_t ttcb_mlp_backward_workspace(int rows, int nin);
int ttcb_mlp_passes_max_features(void);

#ifdef __cplusplus
}
#endif
#endif /* TTCB200_MLP_H */
