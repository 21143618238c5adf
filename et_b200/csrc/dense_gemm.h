// Host-side interface of the dense linear (weights whose zero tiles are cheaper to multiply with than to skip).
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace et {

// Tile width and number of CTAs that share a tile's K range (1: pairs of CTAs, each with the whole range), and the modelled
// clocks of a launch.
struct DensePlan {
    int bn = 0, split = 1;
    double cost = 0;
};
DensePlan dense_plan(int tokens, int N, int K);

// W: [N x K] on the device. kept: bitmap of the kept tiles ([N / 16] rows of whole 32-bit words, a bit per 16 inputs), null when
// none was pruned.
struct DenseWeight {
    const half* W = nullptr;
    const uint32_t* kept = nullptr;
    int N = 0, K = 0;
    CUtensorMap maps[6];   // one per number of weight rows that a CTA may copy at once
};
int dense_map_weight(DenseWeight* w);   // fills in the maps
// bias_given: the bias is the caller's and may be the result of the kernel before.
int dense_run(const DenseWeight& w, const DensePlan& plan, half* Y, const half* X, const half* bias, bool bias_given, int T, int gelu, int* err, cudaStream_t st);

}  // namespace et
