// mlp_train.h - the preconditioner MLP's sizes, packed weights and training
// kernels (mlp_train.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rigidfibers.h"

namespace rf {

constexpr int kMlpIn = RF_MLP_IN, kMlpHid = RF_MLP_HIDDEN, kMlpOut = RF_MLP_OUT;
constexpr int kMlpOutLd = (kMlpOut + 3) / 4 * 4;  // rows of dO start on 16 bytes

// parameter offsets inside the packed weight vector
struct MlpLayout {
    int64_t w1 = 0, b1 = w1 + (int64_t)kMlpHid * kMlpIn, w2 = b1 + kMlpHid, b2 = w2 + (int64_t)kMlpHid * kMlpHid,
            w3 = b2 + kMlpHid, b3 = w3 + (int64_t)kMlpOut * kMlpHid, total = b3 + kMlpOut;
};

// A batch's intermediate results (device; 16-byte aligned)
struct MlpBatch {
    float *h1, *h2, *dO, *dh2, *dh1;   // rows x 256, rows x 256, rows x kMlpOutLd, rows x 256, rows x 256
    float *part;                       // [mlp_slices(rows)][params]
    double *sse;                       // mlp_loss_parts(rows)
};
int mlp_loss_parts(int rows);
int mlp_slices(int rows);   // slices of a batch's weight gradients, not falling with the rows

// G = the gradient of mean (o - Y)^2 over the rows' 225 outputs, *sse += sum
// (o - Y)^2 (device).
cudaError_t mlp_gradient(const MlpBatch &b, const float *W, int rows, const float *X, const float *Y, float *G,
                         double *sse, cudaStream_t st);
// bx, by = rows idx[0..rows) of X, Y
cudaError_t mlp_gather(int rows, const int *idx, const float *X, const float *Y, float *bx, float *by,
                       cudaStream_t st);
cudaError_t mlp_adam(float *W, const float *G, float *m, float *v, float lr, float b1, float b2, float c1, float c2,
                     float eps, cudaStream_t st);

}  // namespace rf
