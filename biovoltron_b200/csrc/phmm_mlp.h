// phmm_mlp.h -- band MLP training interface (kernels in phmm_mlp_train.cu,
// label kernel in phmm_labels.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "phmm_band.h"
#include "phmm_common.h"

namespace bvphmm {

// Flattened FP32 parameters: W1 [kHid][kFeat], b1 [kHid], W2 [kHid][kHid],
// b2 [kHid], W3 [kOut][kHid], b3 [kOut] (weights as [out][in]).
constexpr int kMlpParamCount = kHid * kFeat + kHid + kHid * kHid + kHid + kOut * kHid + kOut;

struct MlpTrainBuffers {
  float* w;      // master weights
  float* g;      // gradient (evaluation)
  float* m;      // Adam moments
  float* v;
  float* X;      // [cap][kFeat] inputs and [cap][2] targets (evaluation; training gathers its rows)
  float* T;
  float* H2;     // [cap][kHid] second hidden layer's activations
  float* O;      // [cap][2] outputs and their gradient
  float* dO;
  float* dH;     // [cap][kHid] gradients of the hidden layers' sums, second and first
  float* dH2;
  float* loss;   // scalar
  float* part1;            // [ceil(cap / 128)][kHid][kFeat] partial products of W1's gradient
  float* part2;            // [ceil(cap / 128)][kHid][kHid] and of W2's
  unsigned int* tc_fail;   // set when a tensor-core product's completion wait gave up
  int cap;
};

// One evaluation of the objective on the n rows of X, T: outputs, loss and, with `backward`, the gradient.
cudaError_t mlp_forward_backward(const MlpTrainBuffers& b, int n, float alpha, bool backward, cudaStream_t st);
// One Adam step (number `step`, from 1) on the n rows idx of feat / targets; adds the loss to *b.loss.
cudaError_t mlp_train_step(const MlpTrainBuffers& b, const __nv_bfloat16* feat, const float* targets, const int32_t* idx,
                           int n, float alpha, int step, float lr, cudaStream_t st);
cudaError_t mlp_export(const float* w, MlpParams* out, cudaStream_t st);

// Label kernel (one warp per pair): the forward rows of every resident warp,
// `stride` floats each, `bytes` in all; pairs whose (R + 1) 3 (H + 2) exceeds
// max_area get no label.  `next`: kLabelClasses work-queue heads, zero.
struct LabelRows {
  long long stride, max_area;
  size_t bytes;
  int blocks;
};
// max_read, max_hap: the longest within the band's limits; longest: the batch's longest read
LabelRows label_rows(int max_read, int longest, int max_hap, int sms, size_t max_bytes);
cudaError_t launch_posterior_spread(const DeviceBatch& b, const Tables* tb, const int32_t* pair_read,
                                    const int32_t* pair_hap, long long n_pairs, float tau, float* fbuf,
                                    const LabelRows& f, int max_hap, unsigned long long* next, int32_t* lo, int32_t* hi,
                                    cudaStream_t st);

}  // namespace bvphmm
