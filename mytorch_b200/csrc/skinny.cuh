// Few-row products y[M,N] = combine(act(norm(x)[M,K] . W[N,K]^T + bias)), M small: the linear
// layers of token-by-token decoding and of tiny batches.
#pragma once
#include "common.cuh"

namespace mt {

struct SkinnyArgs {
  const void* x = nullptr;            // [M, K], row stride ldx
  int64_t ldx = 0;
  int M = 0, K = 0, dtype = 0;
  // up to three weight matrices [n[i], K] (row stride ldw) whose outputs stand side by side in out
  int nseg = 1;
  const void* w[3] = {nullptr, nullptr, nullptr};
  const void* bias[3] = {nullptr, nullptr, nullptr};
  int n[3] = {0, 0, 0};
  int64_t ldw = 0;
  void* out = nullptr;                // [M, sum of n], row stride ldo
  int64_t ldo = 0;
  const void* residual = nullptr;     // added to the result, row stride ldo (may be out itself)
  int act = 0;
  float softcap = 0.f;                // > 0: softcap * tanh(y / softcap) as the last step
  // normalisation of the rows of x in front of the product: 0 none, 1 LayerNorm, 2 RMSNorm
  int norm = 0;
  const void* gamma = nullptr;
  const void* beta = nullptr;
  float eps = 1e-5f;
  // The weights were not written by the kernel just before this one in the stream, so their first
  // pieces may be read before that kernel has finished.
  int early_weights = 0;
};

constexpr int kSkinnyMaxRows = 64;       // half: four 16-row MMA tiles; fp32: chunks of up to 16 rows per block

// How a product is laid out over the chip (gemm_skinny.cu); cost in cycles of the busiest SM.
struct SkinnyShape { int gr, blocks, cluster, kc, its, rounds, ring, x_bytes, nb_bytes; size_t smem; double cost; };
bool skinny_fits(const SkinnyArgs& a, SkinnyShape& shape);      // whether the product can be taken, and how
int skinny_gemm(const SkinnyArgs& a, const SkinnyShape& shape, cudaStream_t st);

}  // namespace mt
