// The NVFP4 GEMM's form on pairs of SMs (gemm_pair.cu), as gemm_tc.cu calls it.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

struct GemmPairArgs {
  const void* wq;        // weights, [N, K/2] or tile-contiguous (w_tiled)
  const void* sfw;       // weight scales, tiled
  const float* tscale;
  const void* xq;        // [tokens * J, K/2]
  const void* sfx;       // activation scales, tiled
  const float* rs;       // [tokens * J]
  const void* residual;  // bf16 [tokens, ldr]
  void* out;
  int ldr, ldo, tokens, J, N, K, epi, w_tiled;
  int pairs;             // pairs of SMs there are
  int parts;             // pairs that share a tile, each a part of K
  int vec;               // rows of a token that are one aligned vector in the output (of SwiGLU half as many results) and the residual: 8, 4 or 1
};

// Launches it with `bn` columns a tile: 32 (one tile of columns only), 64, 128 or 192.
int gemm_pair_launch(const GemmPairArgs& a, int bn, cudaStream_t stream);

// Clusters of `parts` pairs that fit the GPU at a time.
int gemm_pair_clusters(int parts);
