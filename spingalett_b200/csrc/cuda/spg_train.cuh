// spg_train.cuh -- what the files of the training step share: the three products and their arguments.
#pragma once

#include "spg_common.cuh"

// TRAIN_FWD:   C[M][N] = act(A[M][K] . B[N][K]^T + bias[N])        (A = activations, B = weights [out][in])
// TRAIN_DELTA: C[M][N] = (A[M][K] . B[K][N]) * act'(aux[M][N])      (A = delta_{l+1}, B = weights [next][cur])
// TRAIN_GRAD:  C[M][N] = alpha * A[K][M]^T . B[K][N]                 (A = delta [rows][out], B = activations [rows][in]), and, where colsum
//              is not null, colsum[m] = alpha * sum over k of A[k][m] (the bias gradient)
enum { TRAIN_FWD = 0, TRAIN_DELTA = 1, TRAIN_GRAD = 2 };

struct SpgTrainProduct {
    const float *A, *B;
    float *C;
    uint32_t lda, ldb, ldc, M, N, K;
    float alpha;
    const float *bias, *aux;
    uint32_t ldaux;
    int act;
    float *colsum;
};

// whether the tensor-core kernel takes a product: fewer than 148 tiles of 64 x 64
inline bool spg_train_one_kernel(const SpgTrainProduct &p) { return ((p.N + 63) / 64) * ((p.M + 63) / 64) < 148u; }
// two gradients in one launch; SPGK_E_UNSUPPORTED, and nothing launched, for products that are cut differently
int spg_train_two_gradients(const SpgTrainProduct &a, const SpgTrainProduct &b, cudaStream_t s);
// any of the three, on the tensor cores with fp32-level error (spg_train_mma.cu)
int spg_train_product(int mode, const SpgTrainProduct &p, cudaStream_t s);
